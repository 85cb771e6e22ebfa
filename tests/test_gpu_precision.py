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


@pytest.mark.parametrize("p", [4, 8, 12])
def test_leaf_of_many_thousand_bodies(ogx, p):
    """60,000 bodies of one mass in one leaf (the eps floor) act on massless bodies far away, so
    every force goes through the leaf's P2M sums.  A chain of 32 FP32 additions of equal terms is
    off by at most 4.9e-7 (16.5 half ulps), its bodies' masses by 6e-8, the translations by 4e-7
    in the same direction at worst: 1e-6.  One FP32 chain over the whole leaf gave 6.5e-6."""
    rng = np.random.default_rng(p)
    pos = np.concatenate([[0.31, -0.27, 0.44] + 0.02 * (rng.random((60000, 3)) - 0.5),
                          [-0.6, 0.55, -0.3] + 0.8 * (rng.random((3000, 3)) - 0.5)])
    mass = np.concatenate([np.full(60000, 1.0 / 60000), np.zeros(3000)])
    out = {}
    for form in (ogx.PREC_FP64, ogx.PREC_MIXED):
        with ogx.AdaptiveFMM3D(p=p, threshold=64, eps=0.25, precision=form) as s:
            acc, pot = s.compute_accelerations(pos, mass, with_potential=True)
            assert s.stats()["max_leaf_occupancy"] >= 60000
        out[form] = acc[60000:], pot[60000:]
    for a, b in zip(out[ogx.PREC_FP64], out[ogx.PREC_MIXED]):
        assert _rms(a, b) <= 1e-6


@pytest.mark.parametrize("p", [4, 12])
def test_x_lists_of_many_thousand_bodies(ogx, p):
    """Leaves of up to 4,096 bodies round a deep cluster of massless ones: P2L over X lists of
    thousands of bodies, and heavy leaves' M2P the other way.  5e-7: chains of 32 FP32 additions
    and the translations, as above (random terms: 1e-7 measured at p = 4)."""
    rng = np.random.default_rng(p)
    pos = np.concatenate([2.0 * rng.random((120000, 3)) - 1.0,
                          [0.21, -0.13, 0.32] + 0.004 * rng.standard_normal((20000, 3))])
    mass = np.concatenate([np.full(120000, 1.0 / 120000), np.zeros(20000)])
    out = []
    for form in (ogx.PREC_FP64, ogx.PREC_MIXED):
        with ogx.AdaptiveFMM3D(p=p, threshold=4096, precision=form) as s:
            out.append(s.compute_accelerations(pos, mass, with_potential=True))
            assert s.stats()["p2l_evals"] > 100000
    for a, b in zip(*out):
        assert _rms(a[120000:], b[120000:]) <= 5e-7


def _w_lists(ogx, pos, thr):
    """(W member that is a leaf, its centre, one of its bodies, the bodies of the leaves that name it)"""
    with ogx.AdaptiveFMM3D(p=2, threshold=thr) as s:
        s.compute_accelerations(pos, np.ones(len(pos)))
        t = s.tree()
    b, perm = t["boxes"], t["perm"]
    off, idx = t["lists"]["W"]
    named = {}
    for leaf in np.where(b[:, 5] == 1)[0]:
        for w in idx[off[leaf]:off[leaf + 1]]:
            if b[w, 5] == 1:
                named.setdefault(int(w), []).append(leaf)
    for w in sorted(named, key=lambda w: -len(named[w]))[:12]:
        yield t["centers"][w, :3], perm[b[w, 6]], np.concatenate([perm[b[f, 6]:b[f, 6] + b[f, 7]] for f in named[w]])


def test_one_body_through_m2p(ogx):
    """A single massive body at the centre of a W box: its multipole is its mass, and the force on
    the bodies of the leaves that name the box is one M2P evaluation.  Measured 1.32e-7 (mixed) and
    2.4e-16 (FP64) RMS; 2.7e-16 with 1 / r^2 as the square of the inverse root."""
    rng = np.random.default_rng(3)
    pos = np.concatenate([rng.uniform(-1, 1, (6000, 3)), [0.21, -0.13, 0.32] + 0.01 * rng.standard_normal((6000, 3))])
    for form, bound in ((ogx.PREC_MIXED, 1.45e-7), (ogx.PREC_FP64, 2.6e-16)):
        num = den = 0.0
        for centre, body, probes in _w_lists(ogx, pos, 64):
            q, mass = pos.copy(), np.zeros(len(pos))
            q[body], mass[body] = centre, 1.0
            d = centre - q[probes]
            r2 = (d * d).sum(1)
            with ogx.AdaptiveFMM3D(p=4, threshold=64, precision=form) as s:
                e = s.compute_accelerations(q, mass)[probes] - d / r2[:, None] ** 1.5
            num += ((e * e).sum(1) * r2 ** 2).sum()
            den += len(probes)
        assert np.sqrt(num / den) <= bound, (form, np.sqrt(num / den))


def test_spline_kernel_in_fp32(ogx):
    """The mixed form's spline pair in the inner half of the support, against 64 bits: at most
    2.2e-7 with a correctly rounded r (square root, or the residual step); r from the inverse
    square root alone gave 3.0e-7."""
    rng = np.random.default_rng(5)
    h, n = 0.14, 4000
    u = np.sort(rng.uniform(0.02, 0.98, n))
    d = rng.standard_normal((n, 3))
    d *= h * u[:, None] / np.linalg.norm(d, axis=1)[:, None]
    pos, mass = np.concatenate([np.zeros((1, 3)), d]), np.zeros(n + 1)
    mass[0] = 1.0
    u = np.linalg.norm(d, axis=1) / h
    g = np.where(u < 0.5, 32 / 3 + u * u * (32 * u - 38.4),
                 64 / 3 - 48 * u + 38.4 * u * u - 32 / 3 * u ** 3 - 1 / (15 * u ** 3)) / h ** 3
    with ogx.AdaptiveFMM3D(p=2, threshold=4096, eps=h / 2.8, softening=ogx.SOFT_SPLINE, precision=ogx.PREC_MIXED) as s:
        e = np.linalg.norm(s.compute_accelerations(pos, mass)[1:] + g[:, None] * d, axis=1) / (g * h * u)
    assert e[u < 0.5].max() <= 2.5e-7
    assert e[u >= 0.5].max() <= 5e-6      # the outer branch cancels by a factor of up to 40 (3.4e-6 measured)


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
