"""The crease indicator's float pass over the segments against the oracle's walk over all: long
polylines far from the origin, points on, beside and far from them, ends extended and capped.

Neighbour lists do not depend on creases, so the indicator is seen through the shape functions:
one wrong side or cap changes them by the size of the weights; the bar is the FP64 one where creases
truncate supports."""
import numpy as np
import pytest

import curvami_gb300 as cg
from curvami_gb300 import synth
from oracle import Oracle

pytestmark = pytest.mark.gpu


def polylines():
    t = np.linspace(0.0, 1.0, 181)
    return {
        "arc": np.stack([14.0 * np.cos(1.4 * t), 14.0 * np.sin(1.4 * t)], 1),
        "wave": np.stack([1.0 + 18.0 * t, 10.0 + 2.0 * np.sin(9.0 * t)], 1),
        "zigzag": np.stack([2.0 + 16.0 * t, 9.7 + 0.4 * (np.arange(181) % 2)], 1),
    }


@pytest.mark.parametrize("shift", [0.0, 512.0])
@pytest.mark.parametrize("extend", [False, True])
@pytest.mark.parametrize("name", ["arc", "wave", "zigzag"])
def test_against_oracle(name, extend, shift):
    import __graft_entry__ as ge

    ge.build()
    rng = np.random.default_rng(4)
    v = polylines()[name] + shift
    xy = synth.grid_nodes(41, 41, 0.5, 0.1, rng) + shift
    near = v[rng.integers(0, len(v), 300)] + rng.normal(size=(300, 2)) * 10.0 ** rng.uniform(-6, -1, (300, 1))
    pts = np.concatenate([rng.uniform(0.0, 20.0, (1500, 2)) + shift, near])
    pts = pts[((pts > shift) & (pts < 20.0 + shift)).all(1)]
    cut = {"vertices": v, "extend_start": extend, "extend_end": extend, "is_closed": False}
    ctx = cg.Context(0)
    ctx.set_nodes(xy)
    o = Oracle()
    ptr, idx, s = o.frnn(xy, pts, 2.6)
    psi, dpsi, ddpsi, bad, rc = o.rkpm(xy, pts, ptr, idx, s, 2.6, 1, [cut])
    if rc != 0:
        with pytest.raises(cg.CGBError):
            cg.shape_functions(ctx, pts, 2.6, 1, [cut])
        return
    sh = cg.shape_functions(ctx, pts, 2.6, 1, [cut]).download()
    for k, ref in (("psi", psi), ("dpsi", dpsi), ("ddpsi", ddpsi)):
        assert np.abs(sh[k] - ref).max() <= 1e-8 * np.abs(ref).max(), k


@pytest.mark.parametrize("n", [3, 608, 609, 4865])
@pytest.mark.parametrize("name", ["arc", "zigzag"])
def test_lanes_per_point(name, n):
    """32, 4 or one lane per point, by the set's size."""
    import __graft_entry__ as ge

    ge.build()
    rng = np.random.default_rng(n)
    v = polylines()[name][::7]                       # 26 vertices: the last group of segments is part-filled
    xy, pts = synth.grid_nodes(41, 41, 0.5, 0.1, rng), rng.uniform(3.0, 17.0, (n, 2))
    cut = {"vertices": v, "extend_start": True, "extend_end": True, "is_closed": False}
    ctx, o = cg.Context(0), Oracle()
    ctx.set_nodes(xy)
    ptr, idx, s = o.frnn(xy, pts, 2.6)
    psi, dpsi, ddpsi, bad, rc = o.rkpm(xy, pts, ptr, idx, s, 2.6, 1, [cut])
    assert rc == 0
    sh = cg.shape_functions(ctx, pts, 2.6, 1, [cut]).download()
    for k, ref in (("psi", psi), ("dpsi", dpsi), ("ddpsi", ddpsi)):
        assert np.abs(sh[k] - ref).max() <= 1e-8 * np.abs(ref).max(), k
