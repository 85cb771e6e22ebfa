"""How many bits the two forms keep, on inputs where one place shows.  The bars of the other files
(1e-12 for the FP64 form, 5e-6 RMS for the mixed form) leave room for a kernel that holds a value
in fewer bits than it should; the bounds here are about 1.5 times what the kernels show, and below
each stands what a known loss of precision gave."""
import numpy as np
import pytest

import ogx_ic
from helpers import rel_err

pytestmark = pytest.mark.gpu


def _rms(ref, got):
    return float(np.sqrt(((got - ref) ** 2).sum() / (ref ** 2).sum()))


@pytest.mark.parametrize("kind, n, p, thr, eps", [("plummer", 8192, 6, 64, 0.0), ("galaxy", 60000, 8, 64, 0.0), ("galaxy", 60000, 8, 64, 0.05),
                                                  ("cube", 20000, 10, 128, 0.0), ("plummer", 20000, 12, 64, 0.0)])
def test_mixed_form_keeps_its_bits(ogx, kind, n, p, thr, eps):
    """The whole mixed form against the FP64 form: 1.5e-7 to 4e-7 (accelerations, growing with the
    order: the translations' 22 bits) and 0.7e-7 to 1e-7 (potentials) over many sizes."""
    if kind == "plummer":
        pos, _, mass = ogx_ic.plummer(n, seed=n)
    elif kind == "galaxy":
        pos, mass, _ = ogx_ic.disk_bulge(n, seed=n)
    else:
        pos, mass = ogx_ic.uniform_cube(n, seed=n)
    out = []
    for form in (ogx.PREC_FP64, ogx.PREC_MIXED):
        with ogx.AdaptiveFMM3D(p=p, threshold=thr, eps=eps, precision=form) as s:
            out.append(s.compute_accelerations(pos, mass, with_potential=True))
    assert _rms(out[0][0], out[1][0]) <= 6e-7
    assert _rms(out[0][1], out[1][1]) <= 1.5e-7


@pytest.mark.parametrize("p, thr", [(4, 16), (8, 64), (12, 64)])
@pytest.mark.parametrize("form", ["fp64", "fp64rot"])
def test_fp64_forms_keep_their_bits(ogx, oracle, form, p, thr):
    """Both FP64 forms are within 3e-16 of 80-bit arithmetic and the oracle within 9e-16 (RMS)."""
    pos, _, mass = ogx_ic.plummer(6000, seed=p)
    ref, ref_pot = oracle.adaptive_fmm(pos, mass, p=p, thr=thr)
    with ogx.AdaptiveFMM3D(p=p, threshold=thr, precision={"fp64": ogx.PREC_FP64, "fp64rot": ogx.PREC_FP64_ROT}[form]) as s:
        acc, pot = s.compute_accelerations(pos, mass, with_potential=True)
    assert rel_err(ref, acc)[1] <= 2e-15 and _rms(ref_pot, pot) <= 2e-15
