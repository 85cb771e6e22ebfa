"""The work that users of this library have it do, as cases that can be timed and compared.

The calls are the public ones of on-galaxy_b200/ogx.py (the binding of include/ogx.h): force
evaluations on device buffers and on host arrays, leapfrog steps of a resident system, and the
direct sums.  Sizes, orders, leaf capacities and initial conditions are those of the benchmark
configurations and tests:

  * a 16,384-body Plummer sphere, FP64, p = 8, with potentials, against the direct sum;
  * a 262,144-body disk + bulge galaxy, leaf capacities 32 to 128, p from 4 to 12;
  * a two-galaxy merger of a million bodies, mixed form, p = 8;
  * ensembles and served jobs: 8k to 256k bodies (to 1M when served), p in {6, 8, 12}, many
    leapfrog steps of a resident system;
  * the softened merger (eps = 0.05), with Plummer's kernel and with the spline.

A case is {"call", "kind", "n", "p", "leaf", "form", "eps", "soft", "pot", "steps"}:

  call   "device"   compute_accelerations_device on CUDA tensors
         "host"     compute_accelerations on numpy arrays (the ForceSolver3D drop-in's call)
         "steps"    step() of a resident system with captured steps, then download()
         "direct"   DirectSolver3D on CUDA tensors
         "noalloc"  direct_eval_noalloc on numpy arrays
  form   "mixed", "fp64" or "fp64rot" (adaptive FMM only)
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "on-galaxy_b200"))
import ogx  # noqa: E402

DT = 0.001   # eight steps of unsoftened bodies stay comparable between correct implementations


def _case(call, kind, n, p=8, leaf=64, form="mixed", eps=0.0, soft="plummer", pot=False, steps=0, name=None):
    c = {"call": call, "kind": kind, "n": n, "p": p, "leaf": leaf, "form": form, "eps": eps, "soft": soft, "pot": pot,
         "steps": steps}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a few hundred to a few thousand bodies summed directly from host arrays, by a caller
        # that lets no library allocate device memory: the smallest call there is
        _case("noalloc", "plummer", 1000, pot=True, name="direct_noalloc_1000"),
        # the FP64 all-pairs oracle at the size the FMM is checked at
        _case("direct", "plummer", 16384, pot=True, name="direct_plummer_16384"),
        # the accuracy configuration: one FP64 evaluation with potentials, latency-bound
        _case("device", "plummer", 16384, form="fp64", pot=True, name="fp64_plummer_16384_p8"),
        # the FP64 form on the single galaxy, the size at which it is compared with the mixed form
        _case("device", "galaxy", 262144, form="fp64", name="fp64_galaxy_262144_p8"),
        # the third form (rotation M2L) on a mid-sized merger, an odd size
        _case("device", "merger", 100001, form="fp64rot", name="fp64rot_merger_100001_p8"),
        # the smallest ensemble member, p = 6: launches and latency
        _case("device", "plummer", 8192, p=6, name="mixed_plummer_8192_p6"),
        # the single galaxy at low order and small leaves, with potentials
        _case("device", "galaxy", 262144, p=4, leaf=32, pot=True, name="mixed_galaxy_262144_p4_leaf32"),
        # the headline: one evaluation of the million-body merger
        _case("device", "merger", 1000000, name="mixed_merger_1000000_p8"),
        # a served job at the highest order, an odd size
        _case("device", "plummer", 200003, p=12, name="mixed_plummer_200003_p12"),
        # the softened merger without the near/far seam: spline kernel
        _case("device", "merger", 50000, eps=0.05, soft="spline", name="mixed_spline_merger_50000_p8"),
        # an integration job: captured leapfrog steps of a resident system between two downloads
        _case("steps", "galaxy", 30011, p=6, steps=8, name="mixed_steps_galaxy_30011_p6"),
        # the drop-in's call from host arrays
        _case("host", "merger", 120000, name="mixed_host_merger_120000_p8"),
    ]


def _log(rng, lo, hi):
    """Log-uniform whole number, odd ones among them."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["noalloc", "direct", "fp64", "fp64rot", "mixed", "mixed", "mixed", "mixed", "spline", "steps", "host"])
    kind = rng.choice(["plummer", "galaxy", "merger", "cube"])
    pot = rng.random() < 0.3
    leaf = rng.choice([32, 64, 64, 96, 128])
    eps = rng.choice([0.0, 0.0, 0.0, 0.05])
    if what == "noalloc":
        return _case("noalloc", kind, _log(rng, 200, 8000), eps=eps, pot=pot)
    if what == "direct":
        return _case("direct", kind, _log(rng, 2000, 24000), eps=eps, pot=pot)
    if what in ("fp64", "fp64rot"):
        p = rng.choice([4, 6, 8, 10])
        return _case("device", kind, _log(rng, 8192, 262144 if p <= 8 else 131072), p=p, leaf=leaf, form=what, eps=eps, pot=pot)
    if what == "spline":
        return _case("device", kind, _log(rng, 8192, 65536), leaf=leaf, eps=rng.choice([0.02, 0.05]), soft="spline", pot=pot)
    if what == "steps":
        return _case("steps", kind, _log(rng, 8192, 65536), p=rng.choice([6, 8]), leaf=leaf, eps=eps, steps=rng.choice([4, 8]))
    if what == "host":
        return _case("host", kind, _log(rng, 8192, 262144), p=rng.choice([6, 8]), leaf=leaf, eps=eps, pot=pot)
    p = rng.choice([4, 6, 8, 8, 10, 12])
    return _case("device", kind, _log(rng, 8192, 1000000 if p <= 8 else 262144), p=p, leaf=leaf, eps=eps, pot=pot)


# ---------------------------------------------------------------- bodies (made on the GPU)
def _unit(g, n):
    v = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


def _u(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _plummer(g, n):
    """Plummer sphere, scale 1, mass 1, cut at 20; isotropic velocities of the local dispersion."""
    umax = 20.0 ** 3 / (20.0 ** 2 + 1.0) ** 1.5
    u = (_u(g, n) * umax).clamp_min(1e-12)
    r = 1.0 / torch.sqrt(u ** (-2.0 / 3.0) - 1.0)
    pos = r[:, None] * _unit(g, n)
    sig = torch.sqrt(1.0 / (6.0 * torch.sqrt(1.0 + r * r)))
    vel = sig[:, None] * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return pos, vel, torch.full((n,), 1.0 / n, device="cuda", dtype=torch.float64)


def _galaxy(g, n):
    """80% exponential sech^2 disk (scale 1, height 0.1, mass 1), 20% Hernquist bulge (0.2, 0.25)."""
    nb = int(round(0.2 * n))
    nd = n - nb
    cand = -torch.log(_u(g, 4, nd).clamp_min(1e-300) * _u(g, 4, nd).clamp_min(1e-300))   # Gamma(2)
    R = cand[0]
    for k in range(1, 4):
        R = torch.where(R <= 10.0, R, cand[k])
    R = R.clamp_max(10.0)
    ph = 2.0 * math.pi * _u(g, nd)
    z = 0.1 * torch.atanh((2.0 * _u(g, nd) - 1.0) * math.tanh(10.0))
    disk = torch.stack([R * torch.cos(ph), R * torch.sin(ph), z], dim=1)
    s = torch.sqrt(_u(g, nb) * (50.0 / 51.0) ** 2)
    bulge = (0.2 * s / (1.0 - s))[:, None] * _unit(g, nb)
    pos = torch.cat([disk, bulge])
    mass = torch.cat([torch.full((nd,), 1.0 / max(nd, 1), device="cuda", dtype=torch.float64),
                      torch.full((nb,), 0.25 / max(nb, 1), device="cuda", dtype=torch.float64)])
    # circular speed of the enclosed mass
    r = pos.norm(dim=1).clamp_min(1e-3)
    m = 1.0 - (1.0 + r) * torch.exp(-r) + 0.25 * (r / (r + 0.2)) ** 2
    vc = torch.sqrt(m / r)
    rho = torch.sqrt(pos[:, 0] ** 2 + pos[:, 1] ** 2).clamp_min(1e-6)
    vel = torch.stack([-pos[:, 1], pos[:, 0], torch.zeros_like(rho)], dim=1) * (vc / rho)[:, None]
    vel = vel + 0.1 * vc[:, None] * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return pos, vel, mass


def _merger(g, n):
    """Two galaxies at -5 and +5 on x, the second tilted by 30 degrees, relative velocity 0.5."""
    out = []
    c, s = math.cos(math.pi / 6), math.sin(math.pi / 6)
    rot = torch.tensor([[1.0, 0.0, 0.0], [0.0, c, -s], [0.0, s, c]], device="cuda", dtype=torch.float64)
    for k, nk in enumerate((n - n // 2, n // 2)):
        p, v, m = _galaxy(g, nk)
        if k == 1:
            p, v = p @ rot.T, v @ rot.T
        sign = -1.0 if k == 0 else 1.0
        p = p + torch.tensor([5.0 * sign, 0.0, 0.0], device="cuda", dtype=torch.float64)
        v = v + torch.tensor([-0.25 * sign, 0.0, 0.0], device="cuda", dtype=torch.float64)
        out.append((p, v, m))
    return tuple(torch.cat(x) for x in zip(*out))


def _cube(g, n):
    """Uniform cube [-1, 1]^3, masses between 0.5 and 1.5 of the mean, total 1."""
    pos = 2.0 * _u(g, n, 3) - 1.0
    vel = 0.2 * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return pos, vel, (0.5 + _u(g, n)) / n


def _bodies(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    make = {"plummer": _plummer, "galaxy": _galaxy, "merger": _merger, "cube": _cube}[case["kind"]]
    pos, vel, mass = make(g, case["n"])
    return pos.contiguous(), vel.contiguous(), mass.contiguous()


# ---------------------------------------------------------------- the calls
_FORM = {"mixed": ogx.PREC_MIXED, "fp64": ogx.PREC_FP64, "fp64rot": ogx.PREC_FP64_ROT}


def _soft(case):
    return ogx.SOFT_SPLINE if case["soft"] == "spline" else ogx.SOFT_PLUMMER


def prepare(case, seed):
    pos, vel, mass = _bodies(case, seed)
    s = {"case": dict(case)}
    if case["call"] == "noalloc":
        s["pos"], s["mass"] = pos.cpu().numpy(), mass.cpu().numpy()
        return s
    stream = torch.cuda.Stream()
    s["stream"] = stream
    if case["call"] == "direct":
        s["solver"] = ogx.DirectSolver3D(eps=case["eps"], stream=stream.cuda_stream)
    else:
        s["solver"] = ogx.AdaptiveFMM3D(eps=case["eps"], p=case["p"], threshold=case["leaf"], precision=_FORM[case["form"]],
                                        stream=stream.cuda_stream, softening=_soft(case))
    if case["call"] == "steps":
        # a resident system; its steps are captured, as an integration job's are
        s["solver"].upload(pos.cpu().numpy(), vel.cpu().numpy(), mass.cpu().numpy())
        s["solver"].set_tuning(capture_steps=1)
        return s
    acc = torch.empty_like(pos)
    pot = torch.empty_like(mass) if case["pot"] else None
    torch.cuda.synchronize()
    if case["call"] != "direct":
        # a program keeps its solver from one evaluation to the next: this one has evaluated
        # another system of the kind (the mirrored one), so its buffers are there
        s["solver"].compute_accelerations_device(-pos, mass, acc, pot)
        s["solver"].synchronize()
    if case["call"] == "host":
        s["pos"], s["mass"] = pos.cpu().numpy(), mass.cpu().numpy()
    else:
        s.update(pos=pos, mass=mass, acc=acc, potential=pot)
    return s


def run(state):
    c = state["case"]
    if c["call"] == "noalloc":
        out = ogx.direct_eval_noalloc(state["pos"], state["mass"], eps=c["eps"], with_pot=c["pot"])
        return {"acc": out[0], "pot": out[1]} if c["pot"] else {"acc": out}
    s = state["solver"]
    if c["call"] == "host":
        out = s.compute_accelerations(state["pos"], state["mass"], with_potential=c["pot"])
        return {"acc": out[0], "pot": out[1]} if c["pot"] else {"acc": out}
    if c["call"] == "steps":
        s.step(DT, c["steps"])
        pos, vel, acc = s.download()
        return {"pos": pos, "vel": vel, "acc": acc}
    s.compute_accelerations_device(state["pos"], state["mass"], state["acc"], state["potential"])
    return {"acc": state["acc"], "pot": state["potential"]} if c["pot"] else {"acc": state["acc"]}


def work(case):
    """Bytes: positions and masses in, accelerations (and potentials) out.  Operations: the pairs of
    the direct sum at 20 each; for the FMM, what the expansions' passes and the near field take on
    these inputs, from counts on the million-body merger (per body, 9 near pairs per unit of leaf
    capacity, 7 x 64 / leaf M2L translations of 2 (p+1)^4, 15 M2P and 15 P2L evaluations)."""
    n, p, leaf = case["n"], case["p"], case["leaf"]
    bytes_ = n * (32 + 24 + (8 if case["pot"] else 0))
    if case["call"] in ("direct", "noalloc"):
        return {"bytes": bytes_, "flops": 20.0 * n * n}
    k = (p + 1) ** 2
    per_body = 20.0 * min(9.0 * leaf, n) + 7.0 * 64 / leaf * 2 * k * k + 15 * 8.0 * k + 15 * 4.0 * k
    if case["call"] == "steps":
        return {"bytes": n * 2 * 80 * case["steps"], "flops": per_body * n * case["steps"]}
    return {"bytes": bytes_, "flops": per_body * n}


def tolerance(case):
    """Four times what was measured.  FP64: the plain form against the rotation form (other sums of the
    same terms) 2e-15 and at most 2e-14, the direct sum against torch's 5e-15, at most 3e-14.  Mixed form against the
    FP64 form (FP32 pair sums, 22-bit split of the translations): 2e-7 to 6e-7, at most 4e-6; over the
    steps of unsoftened bodies close pairs amplify it."""
    if case["call"] in ("direct", "noalloc") or case["form"] != "mixed":
        return {"rel": 2e-14, "max": 1.1e-13}
    if case["call"] == "steps":
        return {"rel": 1e-5, "max": 5e-4}
    return {"rel": 2.4e-6, "max": 2e-5}


# ---------------------------------------------------------------- 64-bit values
def _spline_gk(r2, h):
    """g(r), k(r) of the cubic spline of Monaghan & Lattanzio in GADGET-2's form, support h."""
    r = torch.sqrt(r2)
    u = r / h
    g1 = (32.0 / 3.0 + u * u * (32.0 * u - 38.4)) / h ** 3
    g2 = (64.0 / 3.0 - 48.0 * u + 38.4 * u * u - 32.0 / 3.0 * u ** 3 - 1.0 / (15.0 * u ** 3)) / h ** 3
    k1 = (2.8 - u * u * (16.0 / 3.0 + u * u * (6.4 * u - 9.6))) / h
    k2 = (3.2 - 1.0 / (15.0 * u) - u * u * (32.0 / 3.0 + u * (-16.0 + u * (9.6 - 32.0 / 15.0 * u)))) / h
    g = torch.where(u < 0.5, g1, torch.where(u < 1.0, g2, 1.0 / (r2 * r)))
    k = torch.where(u < 0.5, k1, torch.where(u < 1.0, k2, 1.0 / r))
    return g, k


def _direct(pos, mass, eps, soft):
    n = pos.shape[0]
    acc, pot = torch.empty_like(pos), torch.empty_like(mass)
    rows = max(1, min(n, (1 << 27) // n))
    for i0 in range(0, n, rows):
        i1 = min(n, i0 + rows)
        d = [pos[None, :, a] - pos[i0:i1, None, a] for a in range(3)]
        r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
        own = torch.arange(i0, i1, device=pos.device)
        r2[own - i0, own] = 1.0
        if soft == "spline" and eps > 0.0:
            g, k = _spline_gk(r2, 2.8 * eps)
        else:
            k = 1.0 / torch.sqrt(r2 + eps * eps)
            g = k * k * k
        m = mass[None, :].expand(i1 - i0, n).clone()
        m[own - i0, own] = 0.0
        g *= m
        for a in range(3):
            acc[i0:i1, a] = (g * d[a]).sum(1)
        pot[i0:i1] = -(k * m).sum(1)
    return acc, pot


def exact(case, seed):
    """The direct sum in 64 bits.  None above 300,000 bodies (minutes), and for an FMM call softened
    with Plummer's kernel: its far field is unsoftened by design, so the direct sum is another value."""
    plummer_fmm = case["call"] not in ("direct", "noalloc") and case["eps"] > 0.0 and case["soft"] == "plummer"
    if case["n"] > 300000 or plummer_fmm:
        return None
    pos, vel, mass = _bodies(case, seed)
    if case["call"] == "steps":
        acc = _direct(pos, mass, case["eps"], case["soft"])[0]
        for _ in range(case["steps"]):
            pos = pos + (vel * DT + acc * (0.5 * DT * DT))
            new = _direct(pos, mass, case["eps"], case["soft"])[0]
            vel = vel + (acc + new) * (0.5 * DT)
            acc = new
        return {"pos": pos, "vel": vel, "acc": acc}
    acc, pot = _direct(pos, mass, case["eps"], case["soft"])
    return {"acc": acc, "pot": pot} if case["pot"] else {"acc": acc}
