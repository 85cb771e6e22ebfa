"""FP64 M2L over work items: every order, trees from one tile cut into 27 slot ranges up to trees
whose tiles are not cut, against the oracle; and a target's result does not depend on its tile."""
import numpy as np
import pytest

import ogx_ic
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", range(1, 13))
def test_every_order_matches_the_oracle(ogx, oracle, p):
    # orders cross every padding of the operand (K mod 4, K mod 8, chunk remainders, column halves);
    # 1e-12: the bar of the FP64 forms (sums of ~1e4 terms at 1.1e-16 each, cancelling)
    pos, _, mass = ogx_ic.plummer(1500, seed=40 + p)
    ref = oracle.adaptive_fmm(pos, mass, p=p, thr=16, with_pot=False)
    for prec in (ogx.PREC_FP64, ogx.PREC_FP64_ROT):
        with ogx.AdaptiveFMM3D(p=p, threshold=16, precision=prec) as s:
            got = s.compute_accelerations(pos, mass)
        assert rel_err(ref, got)[0] <= 1e-12, (p, prec)


@pytest.mark.parametrize("n, thr", [(70, 8), (3001, 16), (40000, 8), (150000, 4)])
def test_every_split_matches_the_oracle(ogx, oracle, n, thr):
    # 70 bodies: a tile or two; 150,000 at leaf 4: above 888 tiles, no split
    pos, _, mass = ogx_ic.plummer(n, seed=n)
    ref = oracle.adaptive_fmm(pos, mass, p=2, thr=thr, with_pot=False)
    for prec in (ogx.PREC_FP64, ogx.PREC_FP64_ROT):
        with ogx.AdaptiveFMM3D(p=2, threshold=thr, precision=prec) as s:
            got = s.compute_accelerations(pos, mass)
        assert rel_err(ref, got)[0] <= 1e-12, (n, prec)


@pytest.mark.parametrize("n", [2000, 30000])
def test_result_does_not_depend_on_the_tile(ogx, n):
    pos, _, mass = ogx_ic.plummer(n, seed=3)
    out = []
    for fill in (128, 32, 96):
        with ogx.AdaptiveFMM3D(p=6, threshold=32, precision=ogx.PREC_FP64) as s:
            s.set_tuning(m2l_tile_targets=fill)
            out.append(s.compute_accelerations(pos, mass))
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("p", [4, 6, 9, 10, 12])
@pytest.mark.parametrize("n", [300, 5000, 60000])
def test_tensor_core_ranges(ogx, p, n):
    # FP64 sums in registers (p <= 8), in TMEM (9, 10), column slices (12); 1 to 27 ranges; with
    # potentials (degree 0).  The batch width changes no bit; 5e-6: the mixed form's bar.
    pos, _, mass = ogx_ic.plummer(n, seed=p)
    with ogx.AdaptiveFMM3D(p=p, threshold=24, precision=ogx.PREC_FP64) as s:
        ref, ref_pot = s.compute_accelerations(pos, mass, with_potential=True)
    out = []
    for fill in (128, 32):
        with ogx.AdaptiveFMM3D(p=p, threshold=24, precision=ogx.PREC_MIXED) as s:
            s.set_tuning(m2l_tile_targets=fill)
            out.append(s.compute_accelerations(pos, mass, with_potential=True))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert rel_err(ref, out[0][0])[1] <= 5e-6
    assert abs(out[0][1] - ref_pot).max() <= 5e-6 * abs(ref_pot).max()
