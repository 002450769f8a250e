"""The elastic hinge beside the FP32 tangent: its blocks must not cost the face part its accuracy.

On a flat regular plate a hinge entry of K is a hundred times the bending entries beside the crease, so
an FP32 sum that holds it rounds the bending part at its size. K of the mixed modes is compared with the
FP64 K per entry, on the scale sqrt(K_ii K_jj) of the face part alone (a bound on the sum of the
magnitudes of an entry's contributions).

Bar: added in FP64, the hinge moves an entry's error by 2^-53 of its value, 2.6e-14 on this scale, so
the largest error is that of the face part alone up to the order of the atomic additions; a factor 2
covers that. The deterministic sums leave nothing to the order: there the hinge's part of the mixed K is
that of the FP64 K to the roundings of the two sums. At most 36 crease points (2 rho / h times the points
per cell) share a pair of nodes, so 80 * 2^-53 of the largest entry."""
import numpy as np
import pytest

import curvami_gb300 as cg
from curvami_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import __graft_entry__ as ge

    ge.build()
    return cg.Context(0)


# quadratic: cells; cubic at rho = 6h: lists above 110, the per-entry tangent
@pytest.mark.parametrize("side, rule, order, rho_factor", [(41, 4, 2, 3.5), (25, 3, 3, 6.0)])
def test_hinge_keeps_face_accuracy(ctx, side, rule, order, rho_factor):
    p = synth.square_plate(side, 0.5, rule, crease="row", Kt=1e-3, kernel=1, rho_factor=rho_factor, order=order, seed=1001)
    asm = cg.PlateModel(p, ctx).asm
    outer, inner = asm.pattern()
    n = 3 * len(p.node_xy)
    col, row = np.repeat(np.arange(n), np.diff(outer)), np.asarray(inner)
    x = np.zeros(n)
    face = asm.assemble(x, cg.TANGENT | cg.DETERMINISTIC)[0].copy()
    both = asm.assemble(x, cg.TANGENT | cg.HINGE | cg.DETERMINISTIC)[0].copy()
    diag = np.zeros(n)
    diag[row[row == col]] = face[row == col]
    scale = np.sqrt(diag[row] * diag[col])
    hinge = both - face
    assert np.abs(hinge).max() > 50.0 * np.median(diag[2::3])
    for mode in (cg.MIXED, cg.MIXED | cg.DETERMINISTIC):
        face32 = asm.assemble(x, cg.TANGENT | mode)[0].copy()
        both32 = asm.assemble(x, cg.TANGENT | cg.HINGE | mode)[0].copy()
        alone = (np.abs(face32 - face) / scale).max()
        assert (np.abs(both32 - both) / scale).max() <= 2.0 * alone, (mode, alone)
        if mode & cg.DETERMINISTIC:
            assert np.abs((both32 - face32) - hinge).max() <= 80.0 * 2.0 ** -53 * np.abs(both).max()
