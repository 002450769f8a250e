"""The neighbour lists and distances, bitwise the oracle's, around 256 candidates per point: the counting
pass keeps the decisions of so many, the filling pass tests the others again. Nodes 0.5 apart, so the 3 x 3
cells of side rho hold about (6 rho)^2: 36, 250, 260, 370 and 580 candidates."""
import numpy as np
import pytest

import curvami_gb300 as cg
from curvami_gb300 import synth
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_node", [False, True])
@pytest.mark.parametrize("rho", [1.0, 2.64, 2.69, 3.2, 4.0])
def test_lists(rho, per_node):
    import __graft_entry__ as ge

    ge.build()
    ctx, o, rng = cg.Context(0), Oracle(), np.random.default_rng(4)
    xy, pts = synth.grid_nodes(41, 41, 0.5, 0.1, rng), rng.uniform(0.0, 20.0, (1025, 2))
    r = rng.uniform(0.95 * rho, 1.1 * rho, len(xy)) if per_node else None
    ctx.set_nodes(xy)
    sh = cg.shape_functions(ctx, pts, rho, 1, [], r).download()
    ptr, idx, s = o.frnn(xy, pts, rho, r)
    assert np.array_equal(sh["ptr"], ptr) and np.array_equal(sh["idx"], idx) and np.array_equal(sh["s"], s)
