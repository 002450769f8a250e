"""Mixed shape functions of one geometry at three scales. The scaled differences are the same, so the
derivatives scale by powers of two; at 2^40 the second derivatives (about 2^-80) and their polynomials
lie below the exponents that the conversions between pairs and doubles treat on the bits, at 2^-40
all are above 1.

Bar: the operations are the same but for parts of pairs below 2^-149, which is 2^-69 of the smallest
scale; a hundred of them are far below one rounding of a double, 2^-52."""
import numpy as np
import pytest

import curvami_gb300 as cg
from curvami_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,kernel", [(1, 0), (2, 0), (2, 1)])
@pytest.mark.parametrize("power", [-40, 40])
def test_powers_of_two(order, kernel, power):
    import __graft_entry__ as ge

    ge.build()
    ctx = cg.Context(0)
    rng = np.random.default_rng(order)
    xy, pts = synth.grid_nodes(21, 21, 0.5, 0.1, rng), rng.uniform(0.0, 10.0, (1000, 2))
    rho = 1.2 if order == 1 else 1.6
    per_node = rng.uniform(0.95 * rho, 1.1 * rho, len(xy))

    def shapes(s):
        ctx.set_nodes(xy * s)
        return cg.shape_functions(ctx, pts * s, rho * s, order, [], per_node * s, kernel, precision="mixed").download()

    a, b, s = shapes(1.0), shapes(2.0 ** power), 2.0 ** power
    assert np.array_equal(a["ptr"], b["ptr"]) and np.array_equal(a["idx"], b["idx"])
    for k, f in (("psi", 1.0), ("dpsi", s), ("ddpsi", s * s)):
        assert np.abs(a[k] - b[k] * f).max() <= 2.0 ** -52 * np.abs(a[k]).max(), k
