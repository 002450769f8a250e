"""The per-entry face tangent against the oracle on lists of the lengths where its pairing of
lanes can go wrong: empty, one, even and odd, around a warp, over 100 neighbours, points that
straddle warps and thread blocks.

Bars: K sums at most 6 * 16 products per value, each rounded a few times (2^-53), so 1e-13 of
the largest value in FP64 (the bar of the FP64 assembly) and 1e-5 with FP32 sums (the bar of
the mixed assembly); F is FP64 in both."""
import numpy as np
import pytest

import curvami_gb300 as cg
from oracle import Oracle

pytestmark = pytest.mark.gpu

LENGTHS = {
    "tiny": [1, 2, 0, 3, 1],
    "warp_edges": [31, 32, 33, 0, 64, 65, 30],
    "many_points": [28, 27, 39, 40] * 20,
    "wide": [113, 112, 160, 159],
}


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__ as ge

    ge.build()
    return cg.Context(0)


def lists(name):
    rng = np.random.default_rng(5)
    n_nodes, counts = 173, LENGTHS[name]
    idx = np.concatenate([rng.permutation(n_nodes)[:n] for n in counts]).astype(np.int32)
    ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    k = len(idx)
    return n_nodes, ptr, idx, rng.normal(size=(k, 2)), rng.normal(size=(k, 3)), rng.uniform(0.5, 1.5, len(counts)), \
        rng.normal(size=3 * n_nodes) * 0.02


@pytest.mark.parametrize("layup", ["isotropic", "unsymmetric"])
@pytest.mark.parametrize("flags", [0, cg.DETERMINISTIC, cg.MIXED, cg.MIXED | cg.DETERMINISTIC])
@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_against_oracle(ctx, name, flags, layup):
    n_nodes, ptr, idx, dpsi, ddpsi, w, x = lists(name)
    o = Oracle()
    if layup == "isotropic":
        A, B, D = cg.abd_isotropic(1.0, 0.3, 0.05)
    else:
        A, B, D = cg.abd_laminate([(1.0, 0.3, 0.3, 0.2, 20.0, 0.03), (1.0, 0.3, 0.3, 0.2, 70.0, 0.02)])
    ctx.set_nodes(np.random.default_rng(1).uniform(size=(n_nodes, 2)))
    asm = cg.NonLinearAssembler(ctx, cg.shape_from_host(ctx, ptr, idx, dpsi, ddpsi), w)
    asm.set_material(A, B, D)
    outer, inner, _, _, mp = o.pattern(n_nodes, ptr, idx, [])
    assert np.array_equal(asm.pattern()[0], outer)
    K, F = asm.assemble(x, cg.TANGENT | flags)
    Ko, Fo = o.update_stiffness(n_nodes, w, ptr, idx, dpsi, ddpsi, outer, mp, x, A, B, D)
    bar = 1e-5 if flags & cg.MIXED else 1e-13
    assert np.abs(K - Ko).max() <= bar * np.abs(Ko).max()
    assert np.abs(F - Fo).max() <= 1e-12 * np.abs(Fo).max()
    if flags & cg.DETERMINISTIC:
        K2, F2 = asm.assemble(x, cg.TANGENT | flags)
        assert np.array_equal(K, K2) and np.array_equal(F, F2)
