"""Leaf far field (L2P, M2P) over the block shapes its rounds can take: leaves of fewer than 16
bodies (whole boxes per round), of more than 64 (several blocks), light and heavy W lists, both
forms, with potentials."""
import pytest

import ogx_ic
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thr", [1, 5, 10, 11, 15, 16, 31, 33, 64, 130])
@pytest.mark.parametrize("p", [1, 4, 5])
def test_block_shapes(ogx, oracle, thr, p):
    n = 600 if thr == 1 else 5000
    pos, _, mass = ogx_ic.plummer(n, seed=thr)
    ref, ref_pot = oracle.adaptive_fmm(pos, mass, p=p, thr=thr)
    with ogx.AdaptiveFMM3D(p=p, threshold=thr, precision=ogx.PREC_FP64) as s:
        got, pot = s.compute_accelerations(pos, mass, with_potential=True)
        alone = s.compute_accelerations(pos, mass)
    # 1e-12: the FP64 form's bar against the reference
    assert rel_err(ref, got)[0] <= 1e-12
    assert abs(pot - ref_pot).max() <= 1e-12 * abs(ref_pot).max()
    assert rel_err(ref, alone)[0] <= 1e-12
    with ogx.AdaptiveFMM3D(p=p, threshold=thr, precision=ogx.PREC_MIXED) as s:
        m, mpot = s.compute_accelerations(pos, mass, with_potential=True)
        malone = s.compute_accelerations(pos, mass)
    # 5e-6 RMS: the mixed form's bar against the FP64 form (its rounding is 2e-7 to 4e-7)
    assert rel_err(ref, m)[1] <= 5e-6 and rel_err(ref, malone)[1] <= 5e-6
    assert abs(mpot - ref_pot).max() <= 5e-6 * abs(ref_pot).max()
