"""Workloads whose time is followed: what a simulation run asks of this framework, through its public entry points.

A run of the real-time SU(3) evolution is a loop of leapfrog steps on a lattice (or on a batch of events of uneven
sizes), with observables measured every few steps, Coulomb gauge fixing of the fields it ends with, and, where
gradients are wanted, the adjoint of the evolution.  The lattices range from the handful of sites of a test to the
128x128x512 production lattice, with extents that are powers of two and extents that are not, in FP64, in FP32 and in
FP32 with 12-real links.

Fields are made with torch from a seed.  "hot": links exp(i 0.3 t.r), E ~ N(0, 0.1^2), currents ~ N(0, 0.02^2) at every
site, as the repository's benchmark fills them.  "collision": the same fields under two Gaussian profiles in z, the
shape of two nuclei with dilute slices (down to ~1e-14 of the peak) around them.

Every case says what it returns; `exact` restates the same in 64-bit torch.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from soerenpragya3dglasma_gb300 import Batch, Lattice

DEV = "cuda"
DT = 0.125
CURRENTS = ("Jp", "Jm", "JpStat", "JmStat")
BATCH_MIX = ((1.0, 1.0, 2.0), (0.75, 0.75, 2.5), (0.5, 0.5, 3.0), (0.9, 0.7, 2.2))


def listed():
    return [
        # the lattice of a unit test or a first try-out: ten steps and their energy, all launches and latency
        {"name": "evolve_fp64_tiny", "kind": "evolve", "nx": 8, "ny": 8, "nz": 16, "az": 1.0, "precision": "fp64",
         "reals": 18, "steps": 10, "fields": "hot"},
        # the small collision the plain method is validated on, advanced from one measurement to the next
        {"name": "evolve_fp64_plain", "kind": "evolve", "nx": 32, "ny": 32, "nz": 128, "az": 1.0, "precision": "fp64",
         "reals": 18, "steps": 10, "fields": "collision"},
        # the production lattice in the default precision
        {"name": "evolve_fp64_production", "kind": "evolve", "nx": 128, "ny": 128, "nz": 512, "az": 1.0,
         "precision": "fp64", "reals": 18, "steps": 2, "fields": "hot"},
        # the production lattice in FP32, one reunitarisation period
        {"name": "evolve_fp32_production", "kind": "evolve", "nx": 128, "ny": 128, "nz": 512, "az": 1.0,
         "precision": "fp32", "reals": 18, "steps": 16, "fields": "hot"},
        # an anisotropic lattice of odd extents in FP32 with 12-real links
        {"name": "evolve_fp32_links12_odd", "kind": "evolve", "nx": 90, "ny": 75, "nz": 201, "az": 0.8,
         "precision": "fp32", "reals": 12, "steps": 16, "fields": "collision"},
        # a sample of independent events of uneven sizes, advanced together from a CUDA graph
        {"name": "evolve_batch_fp32", "kind": "batch", "events": 8, "n": 64, "precision": "fp32", "reals": 18,
         "steps": 16, "fields": "collision"},
        # one measurement of a configuration: energies, Gauss law, energy-momentum map
        {"name": "measure_fp64", "kind": "measure", "nx": 64, "ny": 64, "nz": 256, "az": 1.0, "precision": "fp64",
         "fields": "hot"},
        # the same on an FP32 lattice of extents that are no powers of two
        {"name": "measure_fp32", "kind": "measure", "nx": 96, "ny": 80, "nz": 250, "az": 1.0, "precision": "fp32",
         "fields": "hot"},
        # Coulomb gauge fixing in FP64, extents with factors 3 and 5
        {"name": "gauge_fp64_ragged", "kind": "gauge", "nx": 48, "ny": 40, "nz": 100, "az": 1.0, "mixed": False,
         "iters": 12, "fields": "hot"},
        # Coulomb gauge fixing with FP32 sweeps before the final FP64 transform, a larger power-of-two lattice
        {"name": "gauge_mixed", "kind": "gauge", "nx": 128, "ny": 128, "nz": 256, "az": 1.0, "mixed": True,
         "iters": 40, "fields": "hot"},
        # gradient of the pressure anisotropy after a short FP64 evolution
        {"name": "adjoint_fp64", "kind": "adjoint", "nx": 32, "ny": 32, "nz": 64, "az": 1.0, "precision": "fp64",
         "steps": 20, "fields": "hot"},
        # the same in FP32 on a larger lattice
        {"name": "adjoint_fp32", "kind": "adjoint", "nx": 64, "ny": 64, "nz": 96, "az": 1.0, "precision": "fp32",
         "steps": 40, "fields": "hot"},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def extents(t_lo, t_hi, z_hi, sites):
        """A lattice of at most `sites` sites, with a transverse plane that need not be square."""
        while True:
            nx = log_int(t_lo, t_hi)
            ny = max(t_lo, min(t_hi, int(round(nx * rng.uniform(0.7, 1.3)))))
            nz = max(2 * t_lo, min(z_hi, int(round(nx * rng.uniform(1.5, 4.5)))))
            if nx * ny * nz <= sites:
                return {"nx": nx, "ny": ny, "nz": nz, "az": rng.choice([1.0, 1.0, 0.8])}

    kind = rng.choice(["evolve", "evolve", "evolve", "batch", "measure", "gauge", "adjoint"])
    fields = rng.choice(["hot", "collision"])
    if kind == "evolve":
        precision = rng.choice(["fp64", "fp32"])
        e = extents(8, 128, 512, 2 ** 23)
        big = e["nx"] * e["ny"] * e["nz"] > 2 ** 20
        steps = 16 if precision == "fp32" else rng.choice([1, 2] if big else [4, 10])
        return {"kind": kind, **e, "precision": precision, "reals": rng.choice([18, 12]) if precision == "fp32" else 18,
                "steps": steps, "fields": fields}
    if kind == "batch":
        return {"kind": kind, "events": rng.randint(3, 8), "n": log_int(12, 64), "precision": "fp32",
                "reals": rng.choice([18, 12]), "steps": 16, "fields": fields}
    if kind == "measure":
        return {"kind": kind, **extents(8, 112, 320, 2 ** 21), "precision": rng.choice(["fp64", "fp32"]), "fields": "hot"}
    if kind == "gauge":
        mixed = rng.random() < 0.5
        while True:  # lengths without large prime factors, as a user picks them for the transforms
            e = extents(12, 128 if mixed else 64, 256, 2 ** 22 if mixed else 2 ** 18)
            if all(_smooth(e[k]) for k in ("nx", "ny", "nz")):
                break
        return {"kind": kind, **e, "mixed": mixed, "iters": 40 if mixed else 12, "fields": "hot"}
    precision = rng.choice(["fp64", "fp32"])
    e = extents(8, 64 if precision == "fp32" else 32, 128, 2 ** 19 if precision == "fp32" else 2 ** 16)
    return {"kind": kind, **e, "precision": precision, "steps": 40 if precision == "fp32" else 20, "fields": "hot"}


def _smooth(n):
    for p in (2, 3, 5):
        while n % p == 0:
            n //= p
    return n == 1


# ---- lattices of a case, and their fields ---------------------------------------------------------------------


def _lattices(case):
    """(N, a) of every lattice of the case."""
    if case["kind"] != "batch":
        return [((case["nx"], case["ny"], case["nz"]), (1.0, 1.0, case["az"]))]
    out = []
    for k in range(case["events"]):
        fx, fy, fz = BATCH_MIX[k % len(BATCH_MIX)]
        nx, ny = max(4, int(case["n"] * fx) - k // len(BATCH_MIX)), max(4, int(case["n"] * fy))
        out.append(((nx, ny, max(8, int(nx * fz))), (1.0, 1.0, 1.0)))
    return out


def _herm(v):
    """t^a v^a, (..., 3, 3), with the Gell-Mann matrices over two as t^a."""
    c = 0.5 * v
    s = c[..., 7] / math.sqrt(3.0)
    z = torch.zeros_like(s)
    a01, a02, a12 = (torch.complex(c[..., k], -c[..., k + 1]) for k in (0, 3, 5))
    d = [torch.complex(x, z) for x in (c[..., 2] + s, s - c[..., 2], -2 * s)]
    rows = ((d[0], a01, a02), (a01.conj(), d[1], a12), (a02.conj(), a12.conj(), d[2]))
    return torch.stack([torch.stack(r, dim=-1) for r in rows], dim=-2)


def _mul(*factors):
    """The product of batches of 3x3 matrices, left to right."""
    p = factors[0]
    for f in factors[1:]:
        p = sum(p[..., :, k, None] * f[..., None, k, :] for k in range(3))
    return p


def _expi(c, v):
    """exp(i c t^a v^a) by its Taylor series, as many terms as the largest argument needs."""
    q = 1j * c * _herm(v)
    size = float(torch.linalg.norm(v.detach(), dim=-1).max()) * abs(c)
    terms = 4
    while size ** terms / math.factorial(terms) > 1e-19 and terms < 60:
        terms += 1
    one = torch.eye(3, dtype=torch.complex128, device=DEV)
    x = one + q / terms
    for n in range(terms - 1, 0, -1):
        x = one + _mul(q, x) / n
    return x


def _profile(case, nz):
    """Amplitude per slice."""
    z = torch.arange(nz, device=DEV, dtype=torch.float64)
    if case["fields"] == "hot":
        return torch.ones_like(z)
    w = nz / 16.0
    return torch.exp(-0.5 * ((z - 0.35 * nz) / w) ** 2) + torch.exp(-0.5 * ((z - 0.65 * nz) / w) ** 2)


def _with_ghosts(f):
    return torch.cat([f[:1], f, f[-1:]], dim=0)


def _fields(case, N, seed):
    """U, E and the currents of one lattice in the host layout, ghost slices included, in FP64 (rounded to the
    lattice's precision).  Links in the layout [z+1, y, x, mu, j, i] of the entry points."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    nx, ny, nz = N
    env = _profile(case, nz)[:, None, None, None]

    def normal(*tail):
        return torch.randn((nz, ny, nx) + tail, generator=g, device=DEV, dtype=torch.float64)

    U = torch.empty((nz, ny, nx, 3, 3, 3), dtype=torch.complex128, device=DEV)
    for mu in range(3):
        # 1 + i q, orthonormalised: a link exp(i q) up to second order in q
        v = 0.3 * env * normal(8)
        m = torch.eye(3, dtype=torch.complex128, device=DEV) + 1j * _herm(v)
        r0 = m[..., 0, :] / torch.linalg.norm(m[..., 0, :], dim=-1, keepdim=True)
        r1 = m[..., 1, :] - (r0.conj() * m[..., 1, :]).sum(-1, keepdim=True) * r0
        r1 = r1 / torch.linalg.norm(r1, dim=-1, keepdim=True)
        r2 = torch.linalg.cross(r0, r1, dim=-1).conj()
        U[..., mu, :, :] = torch.stack([r0, r1, r2], dim=-1)  # element (i, j) at [j, i]
        del v, m, r0, r1, r2
    out = {"U": _with_ghosts(U), "E": _with_ghosts(0.1 * env[..., None] * normal(3, 8))}
    del U
    for k in CURRENTS:
        out[k] = _with_ghosts(0.02 * env * normal(8))
    if case.get("precision") == "fp32":
        for k, v in out.items():
            out[k] = v.to(torch.complex64).to(torch.complex128) if v.is_complex() else v.float().double()
    return out


def _upload(lat, fields):
    torch.cuda.synchronize()
    for k, v in fields.items():
        lat.upload_device(k, v.data_ptr())
    lat.synchronize()


def _read(lat, buffers, precision):
    """The lattice's fields into the caller's device buffers, in the lattice's precision."""
    for k, v in buffers.items():
        lat.download_device(k, v.data_ptr())
    if precision == "fp64":
        return dict(buffers)
    return {k: v.to(torch.complex64 if v.is_complex() else torch.float32) for k, v in buffers.items()}


def _numbers(v, precision):
    """Measured numbers in the precision of the fields they were measured on."""
    return np.asarray(v, dtype=np.float64 if precision == "fp64" else np.float32)


# ---- the cases ------------------------------------------------------------------------------------------------


def prepare(case, seed):
    shapes = _lattices(case)
    if case["kind"] == "batch":
        b = Batch([N for N, _ in shapes], [a for _, a in shapes], precision=case["precision"], reunitarize_every=16)
        b.set_step_method("plaquette")
        b.set_link_reals(case["reals"])
        buffers = []
        for k, (N, _) in enumerate(shapes):
            f = _fields(case, N, 1000 * seed + k)
            _upload(b.events[k], f)
            buffers.append({n: torch.empty_like(v) for n, v in f.items()})
        return {"case": case, "batch": b, "buffers": buffers}
    (N, a), = shapes
    precision = case.get("precision", "fp64")
    lat = Lattice(N, a, precision=precision, reunitarize_every=16 if precision == "fp32" else 0)
    f = _fields(case, N, 1000 * seed)
    state = {"case": case, "lat": lat}
    if case["kind"] == "evolve":
        if case["reals"] == 12:
            lat.link_reals = 12
        _upload(lat, f)
        state["buffers"] = {k: torch.empty_like(v) for k, v in f.items()}
        if precision == "fp64":
            state["buffers"]["UOld"] = torch.empty_like(f["U"])
    elif case["kind"] == "measure":
        f["UOld"] = _old_links(f, a, precision)
        _upload(lat, f)
    elif case["kind"] == "gauge":
        _upload(lat, {"U": f["U"], "E": f["E"]})
        state["buffers"] = {"UG": torch.empty_like(f["U"]), "EG": torch.empty_like(f["E"]),
                            "G": torch.empty_like(f["U"][..., 0, :, :]).contiguous()}
    else:
        _upload(lat, f)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        b.step(DT, case["steps"], use_graph=True)
        energy = b.energy()
        return {"energy": _numbers(energy, "fp32"),
                "events": [_read(e, buf, "fp32") for e, buf in zip(b.events, state["buffers"])]}
    lat = state["lat"]
    precision = case.get("precision", "fp64")
    if kind == "evolve":
        # FP64: UOld saved, as the reference's Update leaves it
        lat.step(DT, case["steps"], save_uold=precision == "fp64")
        bulk = lat.bulk()
        return {"bulk": _numbers(bulk, precision), "fields": _read(lat, state["buffers"], precision)}
    if kind == "measure":
        worst, mean, per_slice = lat.gauss(profile=True)
        out = {"bulk": _numbers(lat.bulk(), precision), "gauss": np.array([worst, mean]), "gauss_profile": per_slice,
               "emt": lat.emt_map()}
        if precision == "fp32":
            out["unitarity"] = _numbers(lat.unitarity(), precision)
        return out
    if kind == "gauge":
        lat.gauge_reset()
        log = lat.coulomb_fix(0.08, case["iters"], open_z=True, mixed=case["mixed"], project_zero_mode=case["mixed"])
        precision = "fp32" if case["mixed"] else "fp64"  # the sweeps' arithmetic
        return {"log": _numbers(log, precision), "fields": _read(lat, state["buffers"], precision)}
    value, grads = lat.adjoint(DT, case["steps"], *_slices(case), checkpoint_every=10)
    return {"objective": _numbers(value, precision),
            "grads": {k: v if precision == "fp64" else v.astype(np.float32) for k, v in grads.items()}}


def _slices(case):
    return case["nz"] // 4, case["nz"] - case["nz"] // 4


def work(case):
    """Bytes: each field read once and written once per pass of the algorithm that changes it (a step, a sweep), in the
    precision it is held in, plus what the pass returns.  Flops: the matrix products of the plaquette form (a complex
    3x3 product is 216)."""
    sites = sum(N[0] * N[1] * N[2] for N, _ in _lattices(case))
    real = 8 if case.get("precision", "fp64") == "fp64" else 4
    kind = case["kind"]
    if kind in ("evolve", "batch"):
        links = 3 * case["reals"]
        state = 2 * (links + 24 + 32) * real  # read and written once per step
        # plaquettes 3 x ~2.9 products, 6 rotations and 4 current rotations of ~1.25 products, 4.5 for the links
        return {"bytes": sites * (case["steps"] * state + 110 * (real + 8)), "flops": sites * case["steps"] * 25.7 * 216}
    if kind == "measure":
        # U, UOld, E and the currents once each; energies 6 products, Gauss law 4, map 36 + 4
        return {"bytes": sites * (108 + 24 + 32) * real, "flops": sites * 50 * 216}
    if kind == "gauge":
        r = 4 if case["mixed"] else 8
        # per sweep U and G read, G written (UG may stay on chip), 4 complex planes through two 3D transforms
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": sites * case["iters"] * (54 + 36 + 2 * 8) * r + sites * (54 + 24 + 18) * 16,
                "flops": sites * case["iters"] * (8 * 216 + 2 * 4 * 5 * math.log2(n))}
    # forward, reversed integration and the cotangents' pass: about five steps' work per step
    state = 2 * (54 + 24 + 32) * real
    return {"bytes": sites * (case["steps"] * 3 * state + 56 * 8), "flops": sites * case["steps"] * 4.5 * 25.7 * 216}


# ---- the same in plain 64-bit torch ---------------------------------------------------------------------------


def exact(case, seed):
    kind = case["kind"]
    shapes = _lattices(case)
    sites = sum(N[0] * N[1] * N[2] for N, _ in shapes)
    if kind in ("evolve", "batch"):
        out, energy = [], []
        for k, (N, a) in enumerate(shapes):
            f = _fields(case, N, 1000 * seed + k)
            for _ in range(case["steps"]):
                f = _step(f, a)
            bulk = _bulk(f, a)
            energy.append(bulk[9])
            out.append({"bulk": bulk, "fields": {n: _host(v) for n, v in f.items()}})
        if kind == "batch":
            for o in out:
                o["fields"].pop("UOld")
            return {"energy": torch.stack(energy), "events": [o["fields"] for o in out]}
        if case["precision"] == "fp32":
            out[0]["fields"].pop("UOld")
        return out[0]
    (N, a), = shapes
    f = _fields(case, N, 1000 * seed)
    if kind == "measure":
        f["UOld"] = _old_links(f, a, case["precision"])
        g2, worst = _gauss(f, a)
        out = {"bulk": _bulk(f, a), "gauss": torch.stack([worst, (g2.sum() / (8 * sites)).sqrt()]),
               "gauss_profile": g2 / (N[0] * N[1]), "emt": _emt(f, a)}
        if case["precision"] == "fp32":
            u = _mat(f["U"][1:-1])
            d = torch.linalg.matrix_norm(_mul(u, u.mH) - torch.eye(3, dtype=torch.complex128, device=DEV))
            out["unitarity"] = torch.stack([d.max(), (d.square().sum() / (3 * sites)).sqrt()])
        return out
    if kind == "gauge":
        return _coulomb(f, a, case["iters"], case["mixed"])
    leaf = {k: f[k][1:-1].clone().requires_grad_(True) for k in ("E",) + CURRENTS}
    g = {"U": f["U"], **{k: _with_ghosts(v) for k, v in leaf.items()}}
    for _ in range(case["steps"]):  # each step formed again on the way back: only the states are kept
        g = checkpoint(_step, g, a, use_reentrant=False)
    z0, z1 = _slices(case)
    e, b = _energies(g, a)
    e, b = e[z0:z1].sum(0), b[z0:z1].sum(0)
    value = (e[0] + e[1] - e[2] + b[0] + b[1] - b[2]) / (e[2] + b[2])
    value.backward()
    grads = {}
    for k, v in leaf.items():
        z = torch.zeros_like(v.grad[:1])
        grads[k] = torch.cat([z, v.grad, z], dim=0)
    return {"objective": value.detach(), "grads": grads}


def _mat(u):
    """Stored links [.., j, i] as matrices [.., i, j]."""
    return u.transpose(-1, -2)


def _host(v):
    return v.detach().contiguous()


def _at(f, dx=0, dy=0, dz=0):
    """Values at x + (dx, dy, dz) for the interior sites of a field with ghost slices."""
    n = f.shape[0] - 2
    f = f[1 + dz:1 + dz + n]
    if dx:
        f = torch.roll(f, -dx, dims=2)
    if dy:
        f = torch.roll(f, -dy, dims=1)
    return f


def _unit(mu, s=1):
    return tuple(s if k == mu else 0 for k in range(3))


def _sum(p, q):
    return tuple(i + j for i, j in zip(p, q))


def _retr(m):
    """Re tr(i t^a m), (..., 8)."""
    off = [p for i, j in ((0, 1), (0, 2), (1, 2)) for p in (m[..., i, j].imag + m[..., j, i].imag,
                                                            m[..., i, j].real - m[..., j, i].real)]
    d = [m[..., i, i].imag for i in range(3)]
    last = (d[0] + d[1] - 2 * d[2]) / math.sqrt(3.0)
    return -0.5 * torch.stack(off[:2] + [d[0] - d[1]] + off[2:] + [last], dim=-1)


def _rotate(v, e):
    """2 tr(t^a v (t.e) v^dagger)."""
    return 2 * (_retr(-1j * _mul(v, _herm(e), v.mH)))


def _step(f, a):
    """One leapfrog step: electric field and static currents from U(t), the links in two half steps with the currents'
    update in between."""
    a3 = a[0] * a[1] * a[2]
    U = _mat(_with_ghosts(f["U"][1:-1]))

    def link(mu, d=(0, 0, 0)):
        return _at(U[..., mu, :, :], *d)

    J = {k: f[k] for k in CURRENTS}
    E = []
    for mu in range(3):
        staples = 0
        for nu in range(3):
            if nu == mu:
                continue
            m, n, b = _unit(mu), _unit(nu), _unit(nu, -1)
            up = _mul(link(nu, m), link(mu, n).mH, link(nu).mH)
            down = _mul(link(nu, _sum(m, b)).mH, link(mu, b).mH, link(nu, b))
            staples = staples + (up + down) / a[nu] ** 2
        e = f["E"][1:-1, ..., mu, :] - 2 * DT * a3 / a[mu] ** 2 * _retr(_mul(link(mu), staples))
        if mu == 2:
            e = e - DT / a[2] / math.sqrt(2.0) * (J["Jp"] - J["Jm"])[1:-1]
        E.append(e)
    E = torch.stack(E, dim=-2)
    cj = DT / a[2]
    below = link(2, (0, 0, -1)).mH
    stat = {"JpStat": J["JpStat"][1:-1] - cj * (J["Jp"][1:-1] - _rotate(below, _at(J["Jp"], dz=-1))),
            "JmStat": J["JmStat"][1:-1] + cj * (J["Jm"][1:-1] - _rotate(below, _at(J["Jm"], dz=-1)))}
    stat = {k: _with_ghosts(v) for k, v in stat.items()}
    half, full = [], []
    for mu in range(3):
        x = _expi(-0.5 * DT * a[mu] ** 2 / a3, E[..., mu, :])
        half.append(_mul(x, link(mu)))
        full.append(_mul(x, half[mu]))
    cur = {}
    for k, sign in (("Jp", -1), ("Jm", 1)):
        s = stat[k + "Stat"]
        cur[k] = _with_ghosts(J[k][1:-1] + sign * cj * (_rotate(half[2], _at(s, dz=1)) - s[1:-1]))
    stored = [_with_ghosts(_mat(torch.stack(u, dim=-3))) for u in (full, half)]
    return {"U": stored[0], "E": _with_ghosts(E), **cur, **stat, "UOld": stored[1]}


def _energies(f, a):
    """Per slice: sum E_mu^2 and sum 4 ReTr(1 - P) of the planes yz, zx, xy, times the bulk constants."""
    a3 = a[0] * a[1] * a[2]
    U = _mat(f["U"])
    c = [(a[k] / a3) ** 2 for k in range(3)]
    e = torch.stack([c[k] * f["E"][1:-1, ..., k, :].square().sum((1, 2, 3)) for k in range(3)], dim=-1)
    b = []
    for k, (i, j) in enumerate(((1, 2), (2, 0), (0, 1))):
        p = _mul(_at(U[..., i, :, :]), _at(U[..., j, :, :], *_unit(i)))
        q = _mul(_at(U[..., j, :, :]), _at(U[..., i, :, :], *_unit(j)))
        b.append(c[k] * 4 * (3 - (p * q.conj()).sum((-1, -2)).real).sum((1, 2)))
    return e, torch.stack(b, dim=-1)


def _bulk(f, a):
    e, b = (v.sum(0) for v in _energies(f, a))
    a3 = a[0] * a[1] * a[2]
    c = torch.tensor([(a[k] / a3) ** 2 for k in range(3)], dtype=torch.float64, device=DEV)
    work_done = (f["E"][1:-1, ..., 2, :] * (f["Jp"] - f["Jm"])[1:-1]).sum() / math.sqrt(2.0)
    t = e + b
    zero = torch.zeros_like(work_done)
    tail = [t.sum() / 2] + [t.sum() / 2 - t[k] for k in range(3)] + [e.sum() / 2, b.sum() / 2,
                                                                    a[2] / a3 ** 2 * work_done]
    return torch.cat([e / c, b / c, torch.stack([zero, zero, work_done] + tail)])


def _gauss(f, a):
    """Per slice sum of the squared violation, and its largest component."""
    U = _mat(f["U"])
    total = -(f["JpStat"] + f["JmStat"])[1:-1] / math.sqrt(2.0)
    for mu in range(3):
        b = _unit(mu, -1)
        total = total + f["E"][1:-1, ..., mu, :] - _rotate(_at(U[..., mu, :, :], *b).mH, _at(f["E"][..., mu, :], *b))
    total = total / (a[0] * a[1] * a[2])
    return total.square().sum((1, 2, 3)), total.abs().max()


def _emt(f, a):
    """Transverse averages of T00, TXX, TYY, TZZ, T0X, T0Y, T0Z, TXY, TYZ, TZX per slice."""
    a3 = a[0] * a[1] * a[2]
    q = [a[k] / a3 for k in range(3)]
    U = _mat(f["U"])
    W = _mat(_with_ghosts(f["UOld"][1:-1]))
    B, Bs, E, Es = [], [], [], []
    for k, (m, n) in enumerate(((1, 2), (2, 0), (0, 1))):
        def u(axis, dm, dn):
            return _at(W[..., axis, :, :], *_sum(_unit(m, dm), _unit(n, dn)))

        avg = 0.25 * (_mul(u(m, 0, 0), u(n, 1, 0), u(m, 0, 1).mH, u(n, 0, 0).mH)
                      + _mul(u(n, 0, 0), u(m, -1, 1).mH, u(n, -1, 0).mH, u(m, -1, 0))
                      + _mul(u(n, 0, -1).mH, u(m, 0, -1), u(n, 1, -1), u(m, 0, 0).mH)
                      + _mul(u(m, -1, 0).mH, u(n, -1, -1).mH, u(m, -1, -1), u(n, 0, -1)))
        B.append(q[k] * 2 * _retr(avg))
        Bs.append(q[k] ** 2 * 4 * (3 - avg.diagonal(dim1=-2, dim2=-1).sum(-1).real))
    for mu in range(3):
        b = _unit(mu, -1)
        e, em = f["E"][1:-1, ..., mu, :], _at(f["E"][..., mu, :], *b)
        E.append(q[mu] * 0.5 * (e + _rotate(_at(U[..., mu, :, :], *b).mH, em)))
        Es.append(q[mu] ** 2 * 0.5 * (e.square() + em.square()).sum(-1))
    t = [Es[k] + Bs[k] for k in range(3)]

    def dot(p, r):
        return (p * r).sum(-1)

    t00 = 0.5 * (t[0] + t[1] + t[2])
    cols = [t00] + [t00 - t[k] for k in range(3)]
    cols += [dot(E[i], B[j]) - dot(E[j], B[i]) for i, j in ((1, 2), (2, 0), (0, 1))]
    cols += [dot(E[i], E[j]) + dot(B[i], B[j]) for i, j in ((0, 1), (1, 2), (2, 0))]
    return torch.stack(cols, dim=-1).mean((1, 2))


def _old_links(f, a, precision):
    """Links half a step before U."""
    a3 = a[0] * a[1] * a[2]
    out = torch.empty_like(f["U"])
    for mu in range(3):
        x = _expi(0.5 * DT * a[mu] ** 2 / a3, f["E"][..., mu, :])
        out[..., mu, :, :] = _mat(_mul(x, _mat(f["U"][..., mu, :, :])))
    return out.to(torch.complex64).to(torch.complex128) if precision == "fp32" else out


def _coulomb(f, a, iters, project):
    """The Fourier-accelerated iteration with the open-z functional."""
    U = _mat(f["U"])
    n = U.shape[0] - 2
    shape = U.shape[1:3] + (n,)
    volume = n * shape[0] * shape[1]
    one = torch.eye(3, dtype=torch.complex128, device=DEV)
    G = one.expand((n + 2,) + U.shape[1:3] + (3, 3)).clone()
    c = [1.0 / a[k] ** 2 for k in range(3)]

    def momenta(m, s):
        k = torch.arange(m, device=DEV, dtype=torch.float64)
        return (2 - 2 * torch.cos(2 * math.pi * k / m)) / s ** 2

    p2 = (momenta(n, a[2])[:, None, None] + momenta(shape[0], a[1])[:, None]
          + momenta(shape[1], a[0]))[..., None]
    weight = torch.where(p2 > 0, 1 / (volume * torch.where(p2 > 0, p2, 1.0)), 0.0 if project else 1.0)

    def transform():
        return [_mul(_at(G), _at(U[..., mu, :, :]), _at(G, *_unit(mu)).mH) for mu in range(3)]

    rows = []
    for it in range(iters):
        UG = transform()
        G = _with_ghosts(G[1:-1])
        w = c[0] * (UG[0] + torch.roll(UG[0], 1, dims=2).mH) + c[1] * (UG[1] + torch.roll(UG[1], 1, dims=1).mH)
        up, down = UG[2].clone(), torch.cat([one.expand_as(UG[2][:1]), UG[2][:-1]]).mH
        up[-1] = 0
        w = w + c[2] * (up + down)
        dev = _retr(w)
        lf = w.diagonal(dim1=-2, dim2=-1).sum(-1).real
        upd = torch.fft.ifftn(weight * torch.fft.fftn(dev, dim=(0, 1, 2)), dim=(0, 1, 2), norm="forward").real
        x = _expi(-0.08, upd)
        G[1:-1] = _mul(x.mH, G[1:-1])
        step = (3 - x.diagonal(dim1=-2, dim2=-1).sum(-1)).abs()
        bound = torch.tensor(6.0 * sum(c), dtype=torch.float64, device=DEV)
        rows.append(torch.stack([torch.full_like(bound, it), dev.abs().max(), (dev.square().sum() / (8 * volume)).sqrt(),
                                 step.max(), (step.square().sum() / (8 * volume)).sqrt(),
                                 torch.minimum(lf.min(), bound), lf.sum() / volume]))
    transform()
    G = _with_ghosts(G[1:-1])
    UG = _mat(torch.stack(transform(), dim=-3))
    ghost = one.expand_as(UG[:1]).clone()
    EG = torch.stack([_rotate(_at(G), f["E"][1:-1, ..., mu, :]) for mu in range(3)], dim=-2)
    none = torch.zeros_like(EG[:1])
    return {"log": torch.stack(rows), "fields": {"UG": _host(torch.cat([ghost, UG, ghost])),
                                                 "EG": _host(torch.cat([none, EG, none])), "G": _host(_mat(G))}}
