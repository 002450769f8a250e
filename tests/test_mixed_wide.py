"""The FP32 tangent of wide supports (lists above 110, the per-entry tangent), atomic and deterministic, against
FP64.

A block of K is the sum of m contributions of size t, m up to 9 * 113 here; FP32 forms each with a dozen
roundings, u = 2^-24, independent within a block: an error of 12 u t sqrt(m), 12 u / sqrt(m) = 0.4 u of the
block m t. The largest of 10^6 entries is at 4.9 sigma, 2 u, so the bar is 4 u of the largest entry. Added up in one
float the sum itself is off by about u sqrt(m) / 3 = 10 u, in the same way at every node of a regular
mesh, which Newton paths of such plates do not survive."""
import numpy as np
import pytest

import curvami_gb300 as cg
from curvami_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [cg.MIXED, cg.MIXED | cg.DETERMINISTIC])
def test_wide_supports_sum(mode):
    import __graft_entry__ as ge

    ge.build()
    p = synth.square_plate(31, 0.5, 3, crease="row", Kt=1e-3, kernel=0, rho_factor=6.0, order=3, seed=1001)
    asm = cg.PlateModel(p, cg.Context(0)).asm
    x = np.zeros(3 * len(p.node_xy))
    K = asm.assemble(x, cg.TANGENT | cg.DETERMINISTIC)[0].copy()
    K32 = asm.assemble(x, cg.TANGENT | mode)[0]
    assert np.abs(K32 - K).max() <= 4.0 * 2.0 ** -24 * np.abs(K).max()
