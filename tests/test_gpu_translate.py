"""M2M and L2L over one launch per pass, P2M and P2L over chunks of bodies, pairs in FP64: sizes at
which their loops have remainders, against the oracle."""
import numpy as np
import pytest

import ogx_ic
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p, n, thr", [(1, 9, 1), (2, 400, 2), (3, 20000, 16), (5, 6000, 7), (8, 9000, 40), (12, 3000, 24)])
def test_levels_and_groups_match_the_oracle(ogx, oracle, p, n, thr):
    # one to some hundred groups of 16 parents per level, a dozen levels; 1e-12: the FP64 bar
    pos, _, mass = ogx_ic.plummer(n, seed=7 * p)
    ref = oracle.adaptive_fmm(pos, mass, p=p, thr=thr, with_pot=False)
    with ogx.AdaptiveFMM3D(p=p, threshold=thr) as s:
        assert rel_err(ref, s.compute_accelerations(pos, mass))[0] <= 1e-12
    with ogx.AdaptiveFMM3D(p=p, threshold=thr, precision=ogx.PREC_MIXED) as s:
        assert rel_err(ref, s.compute_accelerations(pos, mass))[1] <= 5e-6   # the mixed form's bar


@pytest.mark.parametrize("thr", [65, 129, 300, 1000])
@pytest.mark.parametrize("p", [4, 10])
def test_leaves_and_lists_of_many_bodies(ogx, oracle, thr, p):
    # P2M in several chunks of 32 or 64 bodies, P2L in several of 128 or 256
    pos, _, mass = ogx_ic.plummer(8000, seed=thr)
    ref, ref_pot = oracle.adaptive_fmm(pos, mass, p=p, thr=thr)
    with ogx.AdaptiveFMM3D(p=p, threshold=thr) as s:
        got, pot = s.compute_accelerations(pos, mass, with_potential=True)
    assert rel_err(ref, got)[0] <= 1e-12
    assert abs(pot - ref_pot).max() <= 1e-12 * abs(ref_pot).max()
    with ogx.AdaptiveFMM3D(p=p, threshold=thr, precision=ogx.PREC_MIXED) as s:
        assert rel_err(ref, s.compute_accelerations(pos, mass))[1] <= 5e-6


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 1000, 2049, 20000])
@pytest.mark.parametrize("eps", [0.0, 0.05])
def test_direct_sum_splits(ogx, oracle, n, eps):
    # 1 to 8 CTAs per 32 targets, whole and partial groups; 1e-12: the direct solver's bar
    pos, mass = ogx_ic.uniform_cube(n, seed=n)
    ref, ref_pot = oracle.direct(pos, mass, eps=eps)
    with ogx.DirectSolver3D(eps=eps) as s:
        got, pot = s.compute_accelerations(pos, mass, with_potential=True)
        alone = s.compute_accelerations(pos, mass)
    assert rel_err(ref, got)[0] <= 1e-12 and rel_err(ref, alone)[0] <= 1e-12
    assert abs(pot - ref_pot).max() <= 1e-12 * max(abs(ref_pot).max(), 1e-300)


def test_pairs_without_a_finite_series(ogx, oracle):
    # coincident bodies, subnormal and overflowing squared distances take the exact pair: the same
    # infinities and NaNs as plain FP64 arithmetic gives, and the other bodies' values
    pos = np.array([[0, 0, 0], [0, 0, 0], [1e-160, 0, 0], [1e-100, 2e-100, 0], [1, 2, 3], [1e200, 0, 0], [-3e155, 1, 2]], float)
    mass = np.array([1.0, 2.0, 3.0, 0.0, 1.0, 1.0, 2.0])
    with np.errstate(all="ignore"):
        d = pos[None] - pos[:, None]
        r2 = (d ** 2).sum(-1)
        ir = 1.0 / np.sqrt(r2)
        w = mass[None] * ir ** 3
        np.fill_diagonal(w, 0.0)
        t = w[..., None] * d
        t[np.arange(7), np.arange(7)] = 0.0
        ref = t.sum(1)
    with ogx.DirectSolver3D() as s:
        got = s.compute_accelerations(pos, mass)
    fin = np.isfinite(ref)
    assert np.array_equal(np.isnan(ref), np.isnan(got))
    assert np.array_equal(fin, np.isfinite(got))
    assert np.allclose(got[fin], ref[fin], rtol=1e-12, atol=0)
