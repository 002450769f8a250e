"""The FP64 moment / solve / value kernels against the oracle: one, two and eight lanes per point (at
the counts where they change on a 152-SM GPU), every order and window, single and per-node radius,
points in the caps of crease ends (the six-jet sums) and beside them, and sets of more points than
one chunk of scratch.

Bars as for the FP64 shape functions: 1e-12 of each array's scale away from the crease (sums of n
products, cond(M) up to a thousand there), 1e-8 where it truncates supports. The cubic basis is held
to the second only: where the plate's corners cut its supports (cond(M) 4e4) the oracle itself is
4e-13 of the scale off the values in extended precision, and these kernels 7e-14."""
import numpy as np
import pytest

import curvami_gb300 as cg
from curvami_gb300 import synth
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__ as ge

    ge.build()
    return cg.Context(0)


def nodes(n=41, h=0.5):
    return synth.grid_nodes(n, n, h, 0.1, np.random.default_rng(3))


def inner_cut(x=10.2, y0=6.0, y1=13.0):
    """A straight cut that ends inside the plate at both ends: half of the points lie in a cap."""
    y = np.linspace(y0, y1, 9)
    return {"vertices": np.stack([np.full(9, x), y], 1), "extend_start": False, "extend_end": False, "is_closed": False}


@pytest.mark.parametrize("cut", [False, True])
@pytest.mark.parametrize("order,rho,kernel", [(1, 1.2, 0), (2, 1.6, 0), (2, 1.6, 1), (3, 2.6, 0)])
@pytest.mark.parametrize("n_gp", [1, 33, 4864, 4865, 19457])
def test_against_oracle(ctx, n_gp, order, rho, kernel, cut):
    rng = np.random.default_rng(n_gp + order)
    xy, pts = nodes(), rng.uniform(0.0, 20.0, (n_gp, 2))
    per_node = rng.uniform(0.95 * rho, 1.1 * rho, len(xy)) if kernel else None
    cuts = [inner_cut()] if cut else []
    ctx.set_nodes(xy)
    sh = cg.shape_functions(ctx, pts, rho, order, cuts, per_node, kernel).download()
    o = Oracle()
    ptr, idx, s = o.frnn(xy, pts, rho, per_node)
    psi, dpsi, ddpsi, _, _ = o.rkpm(xy, pts, ptr, idx, s, rho, order, cuts, per_node, kernel)
    assert np.array_equal(sh["ptr"], ptr) and np.array_equal(sh["idx"], idx) and np.array_equal(sh["s"], s)
    far = np.repeat(np.abs(pts[:, 0] - 10.2) > 1.1 * rho, np.diff(ptr)) if cut else np.ones(len(idx), bool)
    for k, ref in (("psi", psi), ("dpsi", dpsi), ("ddpsi", ddpsi)):
        scale = np.abs(ref).max()
        assert np.abs(sh[k] - ref).max() <= 1e-8 * scale, k
        if far.any() and order < 3:
            assert np.abs(sh[k] - ref)[far].max() <= 1e-12 * scale, k


def test_more_points_than_a_chunk(ctx):
    """1,048,576 points share the scratch: a larger set equals, bitwise, its parts built alone."""
    rng = np.random.default_rng(8)
    xy, pts = nodes(101), rng.uniform(0.0, 50.0, (2**20 + 40000, 2))
    cuts = [inner_cut(25.2, 15.0, 33.0)]
    ctx.set_nodes(xy)
    whole = cg.shape_functions(ctx, pts, 0.9, 1, cuts).download()
    at = 2**20
    for part, g in ((pts[:at], slice(0, at)), (pts[at:], slice(at, len(pts)))):
        sh = cg.shape_functions(ctx, part, 0.9, 1, cuts).download()
        e = slice(whole["ptr"][g.start], whole["ptr"][g.stop])
        for k in ("idx", "s", "psi", "dpsi", "ddpsi"):
            assert np.array_equal(sh[k], whole[k][e]), k
