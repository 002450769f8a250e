"""The tiled face tangent and the deterministic sums against the oracle, where their grouping can go
wrong: a last cell of 1, 15, 16 or 1 + 16 points, cells that share 1, 4, 5 or up to 64 nodes (four
row nodes to an item), points without neighbours, cells whose nodes are too many for a tile beside
cells that have one, a node listed twice by a point; for the sums, node counts around ten
(a block of threads takes ten nodes of F), columns around 14 blocks (one pass of a block of threads)
and up to 260 contributions to a node (128 are fetched at a time).

Bars: K sums m <= 260 * 36 products. A sum of m terms of size t with random signs has a rounding error
of about u t m / sqrt(2) and a largest entry of at least 3 t sqrt(m), so u sqrt(m) / 4 of it: 2e-6 in
FP32 and 4e-15 in FP64. The bars of the mixed and the FP64 assembly, 1e-5 and 1e-13, leave room for the
largest of some thousand entries. F is FP64 in both."""
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


def check(ctx, n_nodes, rows, flags, layup):
    rng = np.random.default_rng(n_nodes + 7 * len(rows))
    ptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int64)
    idx = np.concatenate(rows).astype(np.int32)
    dpsi, ddpsi = rng.normal(size=(len(idx), 2)), rng.normal(size=(len(idx), 3))
    w, x = rng.uniform(0.5, 1.5, len(rows)), rng.normal(size=3 * n_nodes) * 0.02
    if layup == "isotropic":
        A, B, D = cg.abd_isotropic(1.0, 0.3, 0.05)
    else:
        A, B, D = cg.abd_laminate([(1.0, 0.3, 0.3, 0.2, 20.0, 0.03), (1.0, 0.3, 0.3, 0.2, 70.0, 0.02)])
    ctx.set_nodes(rng.uniform(size=(n_nodes, 2)))
    asm = cg.NonLinearAssembler(ctx, cg.shape_from_host(ctx, ptr, idx, dpsi, ddpsi), w)
    asm.set_material(A, B, D)
    o = Oracle()
    outer, _, _, _, mp = o.pattern(n_nodes, ptr, idx, [])
    K, F = asm.assemble(x, cg.TANGENT | flags)
    Ko, Fo = o.update_stiffness(n_nodes, w, ptr, idx, dpsi, ddpsi, outer, mp, x, A, B, D)
    assert np.abs(K - Ko).max() <= (1e-5 if flags & cg.MIXED else 1e-13) * np.abs(Ko).max()
    assert np.abs(F - Fo).max() <= 1e-12 * np.abs(Fo).max()
    if flags & cg.DETERMINISTIC:
        K2, F2 = asm.assemble(x, cg.TANGENT | flags)
        assert np.array_equal(K, K2) and np.array_equal(F, F2)


FLAGS = [cg.DETERMINISTIC, cg.MIXED, cg.MIXED | cg.DETERMINISTIC]


@pytest.mark.parametrize("flags", FLAGS)
@pytest.mark.parametrize("n_gp", [1, 15, 16, 17, 260])
@pytest.mark.parametrize("n_nodes", [1, 4, 5, 10, 11, 14, 15, 29, 60])
def test_small_cells(ctx, n_nodes, n_gp, flags):
    rng = np.random.default_rng(n_gp)
    rows = [rng.permutation(n_nodes)[: n_nodes - g % 2] for g in range(n_gp)]   # one node: every second point is empty
    check(ctx, n_nodes, rows, flags, "isotropic" if n_nodes % 2 else "unsymmetric")


@pytest.mark.parametrize("layup", ["isotropic", "unsymmetric"])
@pytest.mark.parametrize("flags", FLAGS)
def test_tiles_beside_direct_cells(ctx, flags, layup):
    rng = np.random.default_rng(2)
    near = lambda c: c + rng.permutation(40)[:28]             # a cell's points share 40 nodes
    wide = lambda: rng.permutation(300)[:50]                  # 300 nodes in a cell: no tile
    rows = [near(17 * (g // 16)) for g in range(48)] + [wide() for _ in range(16)] + [near(200) for _ in range(16)]
    rows += [np.append(near(100), 105).astype(int) for _ in range(16)]   # some list node 105 twice
    rows += [near(230) for _ in range(5)] + [np.zeros(0, int)] * 20 + [near(3) for _ in range(3)]
    check(ctx, 300, rows, flags, layup)
