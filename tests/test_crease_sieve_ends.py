"""The crease indicator with a short extended last segment, against the oracle's walk over all segments.

The extension of the last segment crosses the first leg of the crease, so near the crossing, in the two wide
sectors, the legs put a point on different sides: the closest segment decides. Points lie 1e-6 to 1e-3
beside the locus of equal distance. With a last segment of 1/1000 to 1/100000 of the others the rounding of its
direction to float moves its extension there by 1e-3 to 1e-1. The bar is that of the other indicator tests: one wrong side
changes the shape functions by the size of the weights."""
import numpy as np
import pytest

import curvami_gb300 as cg
from curvami_gb300 import synth
from oracle import Oracle

pytestmark = pytest.mark.gpu


def crease(last):
    legs = [(1.03, 8.11)] + [(1.03 + 1.61 * k, 8.11 + 0.003 * k) for k in range(1, 11)]
    legs += [(18.23, 9.31), (17.9, 10.7), (16.83, 11.69), (15.0, 11.63), (13.1, 11.51), (11.2, 11.37), (9.31, 11.23)]
    d = np.array([-1.0, -0.553]) / np.hypot(1.0, 0.553)
    return np.array(legs + [tuple(np.array(legs[-1]) + last * d)])


def distances(v, q):
    """Distances of the points q to the segments, the two ends extended: (all but the last, the last)."""
    A, d = v[:-1], np.diff(v, axis=0)
    t = ((q[:, None, :] - A) * d).sum(2) / (d * d).sum(1)
    lo, hi = np.zeros(len(A)), np.ones(len(A))
    lo[0], hi[-1] = -np.inf, np.inf
    r = q[:, None, :] - (A + np.clip(t, lo, hi)[:, :, None] * d)
    r = np.hypot(r[..., 0], r[..., 1])
    return r[:, :-1].min(1), r[:, -1]


def beside_equal_distance(v, rng, count):
    a, b = rng.uniform(0.5, 19.5, (2, 40 * count, 2))
    gap = lambda q: np.subtract(*distances(v, q))
    turn = np.sign(gap(a)) != np.sign(gap(b))
    a, b = a[turn][:count], b[turn][:count]
    s = np.sign(gap(a))
    for _ in range(60):
        m = 0.5 * (a + b)
        same = (np.sign(gap(m)) == s)[:, None]
        a, b = np.where(same, m, a), np.where(same, b, m)
    off = rng.normal(size=a.shape)
    return a + off / np.hypot(*off.T)[:, None] * 10.0 ** rng.uniform(-6, -3, (len(a), 1))


@pytest.mark.parametrize("last", [1.6e-3, 1.6e-4, 1.6e-5])
@pytest.mark.parametrize("count", [500, 3000, 6000])          # 32, 4 and one lane per point
def test_short_extended_end(last, count):
    import __graft_entry__ as ge

    ge.build()
    rng = np.random.default_rng(count)
    v = crease(last)
    xy = synth.grid_nodes(41, 41, 0.5, 0.1, rng)
    pts = beside_equal_distance(v, rng, count)
    assert len(pts) == count
    cut = {"vertices": v, "extend_start": True, "extend_end": True, "is_closed": False}
    ctx, o = cg.Context(0), Oracle()
    ctx.set_nodes(xy)
    ptr, idx, s = o.frnn(xy, pts, 2.6)
    psi, dpsi, ddpsi, bad, rc = o.rkpm(xy, pts, ptr, idx, s, 2.6, 1, [cut])
    if rc != 0:                                               # points whose visible nodes are too few
        pts = pts[np.asarray(bad) == 0]
        assert len(pts) > 0.9 * count
        ptr, idx, s = o.frnn(xy, pts, 2.6)
        psi, dpsi, ddpsi, bad, rc = o.rkpm(xy, pts, ptr, idx, s, 2.6, 1, [cut])
        assert rc == 0
    sh = cg.shape_functions(ctx, pts, 2.6, 1, [cut]).download()
    for k, ref in (("psi", psi), ("dpsi", dpsi), ("ddpsi", ddpsi)):
        assert np.abs(sh[k] - ref).max() <= 1e-8 * np.abs(ref).max(), k
