"""The residual kernel with one to eight lanes per point, at the numbers of points where the
count changes on a 152-SM GPU and beside them, and lists shorter than the lanes.

Bar: F sums about 50 products per node, each a few FP64 roundings of sums over the lists:
1e-13 of its largest value; K (FP64 and FP32 sums) as the assembly's bars."""
import numpy as np
import pytest

import curvami_gb300 as cg
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__ as ge

    ge.build()
    return cg.Context(0)


@pytest.mark.parametrize("flags", [0, cg.TANGENT, cg.TANGENT | cg.MIXED, cg.DETERMINISTIC])
@pytest.mark.parametrize("n_gp", [1, 7, 33, 2432, 2433, 4864, 4865, 9728, 9733])
def test_against_oracle(ctx, n_gp, flags):
    rng = np.random.default_rng(n_gp)
    n_nodes = 211
    counts = rng.integers(1, 12, n_gp)
    ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    idx = np.concatenate([rng.permutation(n_nodes)[:n] for n in counts]).astype(np.int32)
    dpsi, ddpsi = rng.normal(size=(len(idx), 2)), rng.normal(size=(len(idx), 3))
    w, x = rng.uniform(0.5, 1.5, n_gp), rng.normal(size=3 * n_nodes) * 0.02
    o = Oracle()
    A, B, D = cg.abd_laminate([(1.0, 0.3, 0.3, 0.2, 20.0, 0.03), (1.0, 0.3, 0.3, 0.2, 70.0, 0.02)])
    ctx.set_nodes(rng.uniform(size=(n_nodes, 2)))
    asm = cg.NonLinearAssembler(ctx, cg.shape_from_host(ctx, ptr, idx, dpsi, ddpsi), w)
    asm.set_material(A, B, D)
    K, F = asm.assemble(x, flags)
    outer, _, _, _, mp = o.pattern(n_nodes, ptr, idx, [])
    Ko, Fo = o.update_stiffness(n_nodes, w, ptr, idx, dpsi, ddpsi, outer, mp, x, A, B, D)
    assert np.abs(F - Fo).max() <= 1e-13 * np.abs(Fo).max()
    if K is not None:
        assert np.abs(K - Ko).max() <= (1e-5 if flags & cg.MIXED else 1e-13) * np.abs(Ko).max()
