"""Performance cases of the particle-mesh framework: what its users have it do,
through the public Python entry points, over the real range of sizes.

Kinds of work:

* ``force``     PMSolver.compute_forces on host arrays (the stateless drop-in call);
* ``evolve``    upload, KDK steps, download: one evolution of a particle set, in
                both arithmetic forms, with or without per-particle masses, the
                CIC deconvolution and a closing power spectrum;
* ``simulate``  generated initial conditions (Philox field, LPT) into the device
                state, KDK steps, download;
* ``treepm``    the TreePM force method on a handle: a force solve, or KDK steps;
* ``targets``   TreePM short-range forces at a few listed targets, host arrays;
* ``gradient``  loss and d(loss)/d(white noise) through 1LPT and KDK steps, on a
                handle or stateless.

Inputs come from the seed alone: Zel'dovich displacements of a lattice (the
framework's own BBKS table) and, for TreePM, the same with part of the mass
in haloes, as a z = 0 state has. ``exact`` restates the arithmetic in torch in
64 bits (for TreePM with an octree of the same opening criterion).
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

import hyowon_b200 as hb
from hyowon_b200 import adjoint, ic, treepm

DEV = "cuda"
F64 = torch.float64
G_NEWTON = 6.67430e-11 * (1e10 * 1.98847e30) / (3.085677581491367e22 * 1000.0 * 1000.0)
KEYS = ("x", "y", "z", "px", "py", "pz", "ax", "ay", "az")


def listed():
    return [
        # one stateless force call of a small host program (the reference's shipped
        # examples are of this size): latency and launches
        dict(name="force 1e3 mesh 32", kind="force", n=1003, mesh=32, box=50.0,
             precision="fp64", masses=True, deconvolve=False),
        # the smallest benchmark configuration, whole run: many short launches
        dict(name="evolve 32^3 mesh 64 fp64", kind="evolve", n_side=32, mesh=64, box=100.0,
             precision="fp64", masses=False, deconvolve=False, z_start=49.0, steps=32,
             spectrum=False),
        # a mesh and a lattice that are no powers of two, with masses and deconvolution
        dict(name="evolve 75^3 mesh 150 fp64", kind="evolve", n_side=75, mesh=150, box=120.0,
             precision="fp64", masses=True, deconvolve=True, z_start=24.0, steps=16,
             spectrum=False),
        # the accuracy configuration, whole run to z = 0, in the drop-in form ...
        dict(name="evolve 128^3 mesh 256 fp64", kind="evolve", n_side=128, mesh=256, box=256.0,
             precision="fp64", masses=False, deconvolve=False, z_start=49.0, steps=64,
             spectrum=False),
        # ... and in the precision form, closed by its P(k)
        dict(name="evolve 128^3 mesh 256 fp32 P(k)", kind="evolve", n_side=128, mesh=256,
             box=256.0, precision="fp32", masses=False, deconvolve=False, z_start=49.0, steps=64,
             spectrum=True),
        # a production box of ordinary size in the drop-in form, one stretch of steps
        dict(name="evolve 256^3 mesh 512 fp64", kind="evolve", n_side=256, mesh=512, box=500.0,
             precision="fp64", masses=False, deconvolve=False, z_start=49.0, steps=16,
             spectrum=False),
        # the throughput configuration from generated 2LPT initial conditions: the largest
        dict(name="simulate 512^3 mesh 1024 fp32", kind="simulate", n_side=512, mesh=1024,
             box=1000.0, precision="fp32", order=2, z_start=49.0, steps=32),
        # TreePM KDK steps of a clustered set with per-particle masses
        dict(name="treepm 128^3 fp64 2 steps", kind="treepm", n=2097152, mesh=128, box=128.0,
             precision="fp64", masses=True, theta=0.5, steps=2),
        # the TreePM configuration's force on every particle, precision form
        dict(name="treepm 256^3 fp32 force", kind="treepm", n=16777216, mesh=256, box=256.0,
             precision="fp32", masses=False, theta=0.5, steps=0),
        # short-range forces at a sample of particles (an accuracy check of the tree)
        dict(name="targets 4096 of 256^3 fp64", kind="targets", n=16777216, mesh=256, box=256.0,
             precision="fp64", theta=0.5, targets=4096),
        # the differentiable configuration on a handle: one gradient evaluation of an optimiser
        dict(name="gradient 128^3 fp64", kind="gradient", n_side=128, mesh=128, box=256.0,
             precision="fp64", z_start=19.0, steps=16, every=4, handle=True),
        # a small stateless gradient in the precision form, mesh finer than the lattice
        dict(name="gradient 48^3 mesh 96 fp32", kind="gradient", n_side=48, mesh=96, box=100.0,
             precision="fp32", z_start=19.0, steps=8, every=3, handle=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mesh(rng, lo, hi):
    """A mesh side: half the time a power of two, as most users choose."""
    n = _log(rng, lo, hi)
    return n if rng.random() < 0.5 else max(lo, min(hi, 1 << int(round(math.log2(n)))))


def draw(rng):
    kind = rng.choice(["force", "evolve", "evolve", "evolve", "simulate", "treepm", "targets",
                       "gradient"])
    prec = rng.choice(["fp64", "fp32"])
    if kind == "force":
        return dict(kind=kind, n=_log(rng, 300, 1000000), mesh=_mesh(rng, 12, 256),
                    box=round(rng.uniform(20.0, 500.0), 3), precision=prec,
                    masses=prec == "fp64" and rng.random() < 0.5,
                    deconvolve=rng.random() < 0.3)
    if kind == "evolve":
        side = _log(rng, 16, 200)
        return dict(kind=kind, n_side=side, mesh=_mesh(rng, max(12, side // 2), min(384, 2 * side)),
                    box=round(side * rng.uniform(1.0, 3.0), 3), precision=prec,
                    masses=prec == "fp64" and rng.random() < 0.3, deconvolve=rng.random() < 0.3,
                    z_start=round(rng.uniform(9.0, 60.0), 2), steps=_log(rng, 4, 64),
                    spectrum=rng.random() < 0.3)
    if kind == "simulate":
        side = _log(rng, 32, 256)
        return dict(kind=kind, n_side=side, mesh=_mesh(rng, side, 2 * side),
                    box=round(side * rng.uniform(1.0, 3.0), 3), precision=prec,
                    order=rng.choice([1, 2]), z_start=round(rng.uniform(20.0, 60.0), 2),
                    steps=_log(rng, 4, 32))
    if kind == "gradient":
        side = _log(rng, 16, 112)
        # even meshes: the kept potentials of an odd one are not aligned for cuFFT
        return dict(kind=kind, n_side=side, mesh=(_mesh(rng, side, min(158, 2 * side)) + 1) // 2 * 2,
                    box=round(side * rng.uniform(1.0, 3.0), 3), precision=prec, z_start=19.0,
                    steps=_log(rng, 4, 20), every=rng.randint(1, 6), handle=rng.random() < 0.6)
    n = _log(rng, 30000, 3000000)
    side = round(n ** (1.0 / 3.0))
    case = dict(kind=kind, n=n, mesh=_mesh(rng, side, 2 * side), box=float(side),
                precision=prec, theta=rng.choice([0.4, 0.5, 0.7]))
    if kind == "targets":
        return dict(case, targets=_log(rng, 100, min(n, 100000)))
    return dict(case, masses=prec == "fp64" and rng.random() < 0.4, steps=rng.choice([0, 1, 2]))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _rng(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1000003 * int(seed) + salt)


def _modes(n, box):
    """(kx, ky, kz) of the half spectrum and the same with Nyquist zeroed."""
    m = torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=F64)
    k = [2.0 * math.pi / box * m[:, None, None], 2.0 * math.pi / box * m[None, :, None],
         2.0 * math.pi / box * torch.arange(n // 2 + 1, device=DEV, dtype=F64)[None, None, :]]
    d = [v.clone() for v in k]
    if n % 2 == 0:
        d[0][n // 2], d[1][0, n // 2], d[2][0, 0, n // 2] = 0.0, 0.0, 0.0
    return k, d


def _spline(lk, xs, ys, y2):
    hi = torch.searchsorted(xs, lk, right=True).clamp(1, xs.numel() - 1)
    lo = hi - 1
    h = xs[hi] - xs[lo]
    a, b = (xs[hi] - lk) / h, (lk - xs[lo]) / h
    return a * ys[lo] + b * ys[hi] + ((a ** 3 - a) * y2[lo] + (b ** 3 - b) * y2[hi]) * h * h / 6.0


def _displacement(noise, n, box, table):
    """1LPT displacement components (n^3 each) of a white-noise field."""
    xs, ys, y2 = (torch.as_tensor(v, device=DEV, dtype=F64) for v in table)
    k, kd = _modes(n, box)
    k2 = k[0] ** 2 + k[1] ** 2 + k[2] ** 2
    safe = torch.where(k2 > 0, k2, torch.ones_like(k2))
    amp = torch.sqrt(torch.exp(_spline(0.5 * torch.log(safe), xs, ys, y2)) * n ** 3 / box ** 3)
    f = torch.where(k2 > 0, amp / safe, torch.zeros_like(k2))
    w = torch.fft.rfftn(noise.reshape(n, n, n)) * f
    return [torch.fft.irfftn(1j * kd[d] * w, s=(n, n, n)).reshape(-1) for d in range(3)]


def _lattice(n, box):
    q = torch.arange(n, device=DEV, dtype=F64) * (box / n)
    return [v.reshape(-1) for v in torch.meshgrid(q, q, q, indexing="ij")]


def _wrap(x, box):
    w = torch.remainder(x, box)
    return torch.where(w >= box, torch.zeros_like(w), w)


def _lpt_state(case, seed):
    n, box = case["n_side"], case["box"]
    ln_k, ln_p, y2, pf = ic.lpt_table(1.0 / (1.0 + case["z_start"]))
    noise = torch.randn(n ** 3, generator=_rng(seed), device=DEV, dtype=F64)
    psi = _displacement(noise, n, box, (ln_k, ln_p, y2))
    x = [_wrap(q + s, box) for q, s in zip(_lattice(n, box), psi)]
    p = [pf * s for s in psi]
    m = ic.particle_mass(box, n)
    masses = None
    if case.get("masses"):
        masses = m * (0.5 + torch.rand(n ** 3, generator=_rng(seed, 1), device=DEV, dtype=F64))
    return x, p, masses, m


def _clustered_state(case, seed):
    """A z = 0 like set: half the mass in r^-2 haloes of 200 times the mean
    density, the rest on a Zel'dovich-displaced lattice."""
    n, box = case["n"], case["box"]
    g = _rng(seed)
    side = math.ceil(n ** (1.0 / 3.0))
    ln_k, ln_p, y2, _ = ic.lpt_table(0.5)
    noise = torch.randn(side ** 3, generator=g, device=DEV, dtype=F64)
    psi = _displacement(noise, side, box, (ln_k, ln_p, y2))
    pick = torch.randperm(side ** 3, generator=g, device=DEV)[:n]
    x = [(q + s)[pick] for q, s in zip(_lattice(side, box), psi)]
    n_halo = max(1, n // 600)
    size = torch.rand(n_halo, generator=g, device=DEV, dtype=F64).clamp_min(1e-3) ** -0.9
    per = size / size.sum() * (0.5 * n)
    radius = (box / side) * (3.0 * per / (4.0 * math.pi * 200.0)) ** (1.0 / 3.0)
    k = n // 2
    which = torch.searchsorted(torch.cumsum(size / size.sum(), 0),
                               torch.rand(k, generator=g, device=DEV, dtype=F64))
    which = which.clamp_max(n_halo - 1)
    r = radius[which] * torch.rand(k, generator=g, device=DEV, dtype=F64)
    u = torch.randn(3, k, generator=g, device=DEV, dtype=F64)
    u = u / u.norm(dim=0)
    p = []
    for d in range(3):
        x[d][:k] = x[d][-n_halo:][which % n_halo] + r * u[d]
        x[d] = _wrap(x[d], box)
        p.append(150.0 * torch.randn(n, generator=g, device=DEV, dtype=F64))
    m = ic.RHO_CRIT0 * 0.3 * box ** 3 / n
    masses = None
    if case.get("masses"):
        masses = m * (0.5 + torch.rand(n, generator=g, device=DEV, dtype=F64))
    return x, p, masses, m


def _host(t):
    """Pinned host array with the values of a device tensor."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _out(n, keys):
    return {k: torch.empty(n, dtype=F64, pin_memory=True).numpy() for k in keys}


def _schedule(z_start, steps):
    a = 1.0 / (1.0 + z_start)
    return hb.TimeStepper(a, 1.0, math.log(1.0 / a) / steps).factors()


def _tree_lengths(case):
    """(r_s, cutoff, softening) of the TreePM configuration."""
    r_s = 1.25 * case["box"] / case["mesh"]
    return r_s, min(4.5 * r_s, 0.49 * case["box"]), case["box"] / case["n"] ** (1.0 / 3.0) / 30.0


def _tree_factors(case):
    K1, D, K2 = _schedule(49.0, 64)
    return [v[64 - case["steps"]:] for v in (K1, D, K2)]


def _gradient_inputs(case, seed):
    n, N = case["n_side"], case["mesh"]
    noise = torch.randn(n ** 3, generator=_rng(seed), device=DEV, dtype=F64)
    target = 0.5 * torch.randn(N ** 3, generator=_rng(seed, 1), device=DEV, dtype=F64)
    return noise, target


def _force_inputs(case, seed):
    g = _rng(seed)
    n, box = case["n"], case["box"]
    x = torch.rand(3, n, generator=g, device=DEV, dtype=F64) * box
    k = n // 2          # half of it in clumps
    c = torch.rand(3, max(1, n // 100), generator=g, device=DEV, dtype=F64) * box
    at = torch.randint(0, c.shape[1], (k,), generator=g, device=DEV)
    x[:, :k] = _wrap(c[:, at] + 0.02 * box * torch.randn(3, k, generator=g, device=DEV, dtype=F64),
                     box)
    m = ic.RHO_CRIT0 * 0.3 * box ** 3 / n
    masses = m * (0.5 + torch.rand(n, generator=g, device=DEV, dtype=F64)) if case["masses"] else None
    return x, masses, m


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "gradient":
        noise, target = _gradient_inputs(case, seed)
        st["solver"] = None
        if case["handle"]:
            st["solver"] = hb.PMSolver(hb.MeshGeometry(case["box"], case["mesh"]),
                                       hb.PMForceMethod.pure_pm(False), case["precision"])
        st["pm"] = adjoint.DifferentiablePM(case["box"], case["n_side"], case["mesh"],
                                            1.0 / (1.0 + case["z_start"]), case["steps"],
                                            case["precision"], case["every"], solver=st["solver"])
        st["noise"], st["target"] = noise.cpu().numpy(), target.cpu().numpy()
        return st
    if kind == "targets":
        x, _, _, m = _clustered_state(case, seed)
        st["x"], st["m"] = [v.cpu().numpy() for v in x], m
        pick = torch.randperm(case["n"], generator=_rng(seed, 2), device=DEV)[:case["targets"]]
        st["targets"] = pick.cpu().numpy().astype(np.uint32)
        return st
    method = hb.PMForceMethod.pure_pm(bool(case.get("deconvolve")))
    if kind == "treepm":
        method = hb.PMForceMethod.treepm_long_range(_tree_lengths(case)[0])
    s = hb.PMSolver(hb.MeshGeometry(case["box"], case["mesh"]), method, case["precision"])
    st["s"] = s
    if kind == "force":
        x, masses, m = _force_inputs(case, seed)
        st["x"] = [v.cpu().numpy() for v in x]
        st["masses"] = None if masses is None else masses.cpu().numpy()
        st["m"] = m
        st["acc"] = [np.zeros(case["n"]) for _ in range(3)]
        return st
    if kind == "simulate":
        a = 1.0 / (1.0 + case["z_start"])
        st["params"] = ic.ICParams(case["n_side"], case["box"], 1 + int(seed), a,
                                   lpt_order=case["order"])
        st["power"] = ic.power_table(st["params"], ic.start_spectrum(a))
        st["m"] = ic.particle_mass(case["box"], case["n_side"])
        st["factors"] = [v[:case["steps"]] for v in _schedule(case["z_start"], 2 * case["steps"])]
        st["out"] = _out(case["n_side"] ** 3, KEYS[:6])
        return st
    if kind == "treepm":
        x, p, masses, m = _clustered_state(case, seed)
        _, cut, eps = _tree_lengths(case)
        s.set_treepm_short_range(case["theta"], eps, cut)
        st["factors"] = _tree_factors(case)
        keys = KEYS if case["steps"] else KEYS[6:]
    else:
        x, p, masses, m = _lpt_state(case, seed)
        st["factors"] = _schedule(case["z_start"], case["steps"])
        keys = KEYS
    st["x"], st["p"] = [_host(v) for v in x], [_host(v) for v in p]
    st["masses"] = None if masses is None else _host(masses)
    st["m"] = None if masses is not None else m
    st["out"] = _out(x[0].numel(), keys)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "gradient":
        loss, grad = st["pm"].loss_and_grad(st["noise"], st["target"])
        return {"loss": loss, "grad": grad}
    if kind == "targets":
        r_s, cut, eps = _tree_lengths(case)
        ax, ay, az, _ = treepm.short_range_forces(case["box"], *st["x"], st["m"], st["targets"],
                                                  r_s, cut, eps, case["theta"], case["precision"])
        return {"ax": ax, "ay": ay, "az": az}
    s = st["s"]
    if kind == "force":
        for a in st["acc"]:
            a.fill(0.0)
        s.compute_forces(*st["x"], st["masses"], None if st["masses"] is not None else st["m"],
                         *st["acc"])
        return list(st["acc"])
    if kind == "simulate":
        s.generate_ics(st["params"], st["power"], st["m"])
        drift = s.run(*st["factors"])
        return dict(s.download(out=st["out"]), drift=drift)
    s.upload(*st["x"], *st["p"], masses=st["masses"], uniform_mass=st["m"])
    if kind == "treepm" and case["steps"] == 0:
        s.solve_forces()
        return s.download(out=st["out"])
    drift = s.run(*st["factors"])
    r = dict(s.download(out=st["out"]), drift=drift)
    if case.get("spectrum"):
        r["spectrum"] = s.power_spectrum(24)
    return r


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------
def _step_bytes(case, n):
    """One force solve and KDK update: each particle field and mesh pass once."""
    b = 8 if case["precision"] == "fp64" else 4
    return n * 15 * b + case["mesh"] ** 3 * 6 * b


def work(case):
    kind, N = case["kind"], case["mesh"]
    n = case["n"] if "n" in case else case["n_side"] ** 3
    fft = 5.0 * N ** 3 * math.log2(N ** 3)          # both transforms of a real field
    solve = fft + 200.0 * n
    if kind == "force":
        return {"bytes": 64.0 * n + _step_bytes(case, n), "flops": solve}
    if kind == "gradient":
        steps = case["steps"] + 1
        return {"bytes": 24.0 * n + 8.0 * N ** 3 + 3.0 * steps * _step_bytes(case, n),
                "flops": 3.0 * steps * solve}
    # short range: a few hundred pair interactions of about 30 operations a target
    if kind == "targets":
        return {"bytes": 24.0 * n + 28.0 * case["targets"], "flops": 2.0e4 * case["targets"]}
    if kind == "treepm":
        solves = case["steps"] + 1
        return {"bytes": 120.0 * n + solves * (_step_bytes(case, n) + 48.0 * n),
                "flops": solves * (2.0e4 * n + 2.0 * solve)}
    solves = case["steps"] + 1
    return {"bytes": 96.0 * n + solves * _step_bytes(case, n), "flops": solves * solve}


def tolerance(case):
    """Relative differences between correct implementations: about four times
    the distance to `exact` where the two differ in summation order only. An
    evolution amplifies rounding (more so in a small box), and a tree target
    whose opening decision lies on the edge can take the other branch."""
    fp64 = case["precision"] == "fp64"
    if case["kind"] == "gradient":
        return {"rel": 1e-10, "max": 1e-6} if fp64 else {"rel": 4e-3, "max": 0.4}
    if case["kind"] in ("treepm", "targets"):
        return {"rel": 1e-9, "max": 1e-5} if fp64 else {"rel": 1e-4, "max": 1e-2}
    return {"rel": 5e-11, "max": 1e-7} if fp64 else {"rel": 4e-4, "max": 4e-2}


# --------------------------------------------------------------------------
# the same in 64 bits, plain torch
# --------------------------------------------------------------------------
def _corners(x, box, N):
    """Flat cell index and weight of the 8 CIC corners."""
    i, f = [], []
    for v in x:
        s = (v / (box / N)).clamp(max=math.nextafter(float(N), 0.0))
        b = torch.floor(s.detach())
        i.append(b.long())
        f.append(s - b)
    for ox in (0, 1):
        for oy in (0, 1):
            for oz in (0, 1):
                cell = ((((i[0] + ox) % N) * N + (i[1] + oy) % N) * N + (i[2] + oz) % N)
                w = ((f[0] if ox else 1.0 - f[0]) * (f[1] if oy else 1.0 - f[1])
                     * (f[2] if oz else 1.0 - f[2]))
                yield cell, w


def _deposit(x, box, N, m):
    mesh = torch.zeros(N ** 3, device=DEV, dtype=F64)
    for cell, w in _corners(x, box, N):
        mesh = mesh.index_add(0, cell, m * w)
    return mesh.reshape(N, N, N)


def _window(N):
    m = torch.fft.fftfreq(N, 1.0 / N, device=DEV, dtype=F64)
    w = torch.sinc(m / N) ** 2
    return w[:, None, None] * w[None, :, None] * w[None, None, :N // 2 + 1]


def _pm_force(x, box, N, m, deconvolve=False, r_s=None):
    dx = box / N
    d = torch.fft.rfftn(_deposit(x, box, N, m)) * (4.0 * math.pi * G_NEWTON / dx ** 3)
    if r_s is None:
        s = torch.sin(math.pi * torch.fft.fftfreq(N, 1.0 / N, device=DEV, dtype=F64) / N)
        s = -4.0 / dx ** 2 * s * s
        lap = s[:, None, None] + s[None, :, None] + s[None, None, :N // 2 + 1]
    else:
        k, kd = _modes(N, box)
        lap = -(k[0] ** 2 + k[1] ** 2 + k[2] ** 2)
    lap[0, 0, 0] = 1.0
    f = 1.0 / lap
    f[0, 0, 0] = 0.0
    if r_s is not None:
        f = f * torch.exp(lap * r_s * r_s)
        f[0, 0, 0] = 0.0
    if deconvolve or r_s is not None:
        f = f / _window(N) ** 2
    d = d * f
    if r_s is None:
        phi = torch.fft.irfftn(d, s=(N, N, N))
        g = [-(torch.roll(phi, -1, a) - torch.roll(phi, 1, a)) / (2.0 * dx) for a in range(3)]
    else:
        g = [torch.fft.irfftn(-1j * kd[a] * d, s=(N, N, N)) for a in range(3)]
    acc = [torch.zeros_like(x[0]) for _ in range(3)]
    for cell, w in _corners(x, box, N):
        for a in range(3):
            acc[a] = acc[a] + w * g[a].reshape(-1)[cell]
    return acc


def _short_factor(r2, eps2, r_s):
    q = torch.sqrt(r2) / r_s
    isp = 1.0 / math.sqrt(math.pi)
    q2 = q * q
    series = 1.0 / ((r2 + eps2) * torch.sqrt(r2 + eps2)) - isp / r_s ** 3 * (
        1.0 / 6.0 + q2 * (-1.0 / 40.0 + q2 * (1.0 / 448.0 + q2 * (-1.0 / 6912.0 + q2 / 135168.0))))
    ms = torch.special.erfc(0.5 * q) + q * isp * torch.exp(-0.25 * q2)
    far = (torch.expm1(-1.5 * torch.log1p(eps2 / r2)) + ms) / (r2 * torch.sqrt(r2))
    return torch.where(q < 0.05, series, far)


def _min_image(d, box):
    return torch.where(d >= 0.5 * box, d - box, torch.where(d < -0.5 * box, d + box, d))


def _spread(v):
    for s, k in ((32, 0x1f00000000ffff), (16, 0x1f0000ff0000ff), (8, 0x100f00f00f00f00f),
                 (4, 0x10c30c30c30c30c3), (2, 0x1249249249249249)):
        v = (v | (v << s)) & k
    return v


def _tree_force(x, box, m, r_s, cut, eps, theta, targets=None):
    """Short-range sum over an octree with the framework's opening criterion,
    all (target, node) pairs of a level at a time."""
    n = x[0].numel()
    m = torch.full((n,), m, device=DEV, dtype=F64) if isinstance(m, float) else m
    q = [torch.floor(v / box * 2097152.0).clamp(0, 2097151).long() for v in x]
    key, order = torch.sort((_spread(q[0]) << 2) | (_spread(q[1]) << 1) | _spread(q[2]))
    src = torch.stack([v[order] for v in x])
    ms = m[order]
    slot = torch.empty(n, dtype=torch.long, device=DEV)
    slot[order] = torch.arange(n, device=DEV)
    t_all = slot if targets is None else slot[targets]
    levels = []
    for level in range(22):
        pre, run, cnt = torch.unique_consecutive(key >> (3 * (21 - level)), return_inverse=True,
                                                 return_counts=True)
        start = torch.cumsum(cnt, 0) - cnt
        mass = torch.zeros(pre.numel(), device=DEV, dtype=F64).index_add_(0, run, ms)
        com = torch.stack([torch.zeros_like(mass).index_add_(0, run, ms * src[a]) for a in range(3)])
        cell = torch.zeros(3, pre.numel(), dtype=torch.long, device=DEV)
        for b in range(level):
            o = (pre >> (3 * (level - 1 - b))) & 7
            cell = (cell << 1) | torch.stack([o >> 2, (o >> 1) & 1, o & 1])
        side = box / 2.0 ** level
        centre = (cell.double() + 0.5) * side
        com = com / mass
        need = side / theta + (com - centre).abs().sum(0)
        levels.append(dict(pre=pre, run=run, cnt=cnt, start=start, mass=mass, com=com,
                           centre=centre, half=0.5 * side, open2=need * need))
        if int(cnt.max()) == 1:
            break
    acc = torch.zeros(3, n, device=DEV, dtype=F64)

    def add(t, d, r2, w):
        f = G_NEWTON * w * _short_factor(r2, eps * eps, r_s)
        for a in range(3):
            acc[a].index_add_(0, t, f * d[a])

    for t0 in torch.split(t_all, 65536):
        t, node = t0, torch.zeros_like(t0)
        for level, lv in enumerate(levels):
            h = lv["half"]
            d = _min_image(lv["centre"][:, node] - src[:, t], box).abs()
            if h >= 0.25 * box:
                keep, inside = torch.ones_like(t, dtype=torch.bool), torch.zeros_like(t, dtype=torch.bool)
            else:
                keep = ((d - h).clamp_min(0.0) ** 2).sum(0) < cut * cut
                inside = ((d + h) ** 2).sum(0) < cut * cut
            t, node, inside = t[keep], node[keep], inside[keep]
            leaf = (lv["cnt"][node] == 1) | (level == 21)
            tl, nl = t[leaf], node[leaf]
            c = lv["cnt"][nl]
            tp = torch.repeat_interleave(tl, c)
            first = torch.repeat_interleave(lv["start"][nl] - (torch.cumsum(c, 0) - c), c)
            sp = first + torch.arange(tp.numel(), device=DEV)
            dv = _min_image(src[:, sp] - src[:, tp], box)
            r2 = (dv * dv).sum(0)
            ok = (r2 < cut * cut) & (r2 > 0.0) & (sp != tp)
            add(tp[ok], dv[:, ok], r2[ok], ms[sp[ok]])
            t, node, inside = t[~leaf], node[~leaf], inside[~leaf]
            dv = _min_image(lv["com"][:, node] - src[:, t], box)
            r2 = (dv * dv).sum(0)
            take = inside & (r2 > lv["open2"][node]) & ((key[t] >> (3 * (21 - level))) != lv["pre"][node])
            add(t[take], dv[:, take], r2[take], lv["mass"][node[take]])
            t, node = t[~take], node[~take]
            if t.numel() == 0 or level + 1 == len(levels):
                break
            nxt = levels[level + 1]["run"]
            first = nxt[lv["start"][node]]
            c = nxt[lv["start"][node] + lv["cnt"][node] - 1] - first + 1
            t = torch.repeat_interleave(t, c)
            node = torch.repeat_interleave(first - (torch.cumsum(c, 0) - c), c) \
                + torch.arange(t.numel(), device=DEV)
    return [acc[a][t_all] for a in range(3)]


def _kdk(x, p, force, factors, box):
    a = force(x)
    drift = []
    for K1, D, K2 in zip(*factors):
        p = [v + g * K1 for v, g in zip(p, a)]
        drift.append(float((D * D * (p[0] ** 2 + p[1] ** 2 + p[2] ** 2)).max().sqrt()))
        x = [_wrap(v + D * w, box) for v, w in zip(x, p)]
        a = force(x)
        p = [v + g * K2 for v, g in zip(p, a)]
    return x, p, a, np.array(drift)


def _spectrum(x, box, N, bins):
    n = x[0].numel()
    d = _deposit(x, box, N, 1.0) / (n / N ** 3) - 1.0
    d = torch.fft.rfftn(d) / N ** 3
    d[0, 0, 0] = 0.0
    k, _ = _modes(N, box)
    km = torch.sqrt(k[0] ** 2 + k[1] ** 2 + k[2] ** 2)
    k_max = math.pi * N / box
    lo = 2.0 * math.pi / box
    edges = torch.as_tensor([lo * (k_max / lo) ** (i / bins) for i in range(bins + 1)], device=DEV, dtype=F64)
    edges[0], edges[-1] = lo, k_max
    b = torch.searchsorted(edges, km * (1.0 + 1e-14), right=True) - 1
    raw = box ** 3 * d.abs() ** 2
    dec = 1.0 / _window(N) ** 2
    mult = torch.full_like(km, 2.0)
    mult[:, :, 0] = 1.0
    if N % 2 == 0:
        mult[:, :, N // 2] = 1.0
    sel = (b >= 0) & (b < bins) & (km > 0) & (km <= k_max)
    cnt = torch.zeros(bins, device=DEV, dtype=F64).index_add_(0, b[sel], mult[sel])

    def mean(v):
        s = torch.zeros(bins, device=DEV, dtype=F64).index_add_(0, b[sel], (v * mult)[sel])
        return (s / cnt.clamp_min(1.0)).cpu().numpy()

    return {"k_low": edges[:-1].cpu().numpy(), "k_mean": mean(km), "k_high": edges[1:].cpu().numpy(),
            "p_raw": mean(raw), "p_corrected": mean(raw * dec),
            "mean_cic_power_deconvolution_factor": mean(dec),
            "shot_noise_reference": np.full(bins, box ** 3 / n), "mode_count": None}


def exact(case, seed):
    kind, box, N = case["kind"], case["box"], case["mesh"]
    if kind == "simulate":
        return None     # the Philox per-mode generator has no plain torch counterpart
    if kind == "gradient":
        return _exact_gradient(case, seed)
    if kind == "force":
        x, masses, m = _force_inputs(case, seed)
        a = _pm_force(list(x), box, N, m if masses is None else masses, case["deconvolve"])
        return [v.cpu().numpy() for v in a]
    if kind in ("treepm", "targets"):
        x, p, masses, m = _clustered_state(case, seed)
        r_s, cut, eps = _tree_lengths(case)
        m = float(m) if masses is None else masses
        if kind == "targets":
            pick = torch.randperm(case["n"], generator=_rng(seed, 2), device=DEV)[:case["targets"]]
            a = _tree_force(x, box, m, r_s, cut, eps, case["theta"], pick)
            return {k: v.cpu().numpy() for k, v in zip(KEYS[6:], a)}
        if (case["steps"] + 1) * case["n"] > 2e7:
            return None

        def force(y):
            long = _pm_force(y, box, N, m, r_s=r_s)
            return [u + v for u, v in zip(long, _tree_force(y, box, m, r_s, cut, eps, case["theta"]))]

        if case["steps"] == 0:
            return {k: v.cpu().numpy() for k, v in zip(KEYS[6:], force(x))}
        x, p, a, drift = _kdk(x, p, force, _tree_factors(case), box)
    else:
        x, p, masses, m = _lpt_state(case, seed)
        m = m if masses is None else masses
        x, p, a, drift = _kdk(x, p, lambda y: _pm_force(y, box, N, m, case["deconvolve"]),
                              _schedule(case["z_start"], case["steps"]), box)
    r = {k: v.cpu().numpy() for k, v in zip(KEYS, x + p + a)}
    r["drift"] = drift
    if case.get("spectrum"):
        r["spectrum"] = None if case.get("masses") else _spectrum(x, box, N, 24)
    return r


def _exact_gradient(case, seed):
    n, N, box = case["n_side"], case["mesh"], case["box"]
    ln_k, ln_p, y2, pf = ic.lpt_table(1.0 / (1.0 + case["z_start"]))
    noise, target = _gradient_inputs(case, seed)
    noise.requires_grad_(True)
    m = ic.particle_mass(box, n)
    factors = _schedule(case["z_start"], case["steps"])
    psi = _displacement(noise, n, box, (ln_k, ln_p, y2))
    x = [_wrap(q + s, box) for q, s in zip(_lattice(n, box), psi)]
    p = [pf * s for s in psi]

    def step(K1, D, K2, *s):
        x, p, a = list(s[:3]), list(s[3:6]), list(s[6:])
        p = [v + g * K1 for v, g in zip(p, a)]
        x = [_wrap(v + D * w, box) for v, w in zip(x, p)]
        a = _pm_force(x, box, N, m)
        p = [v + g * K2 for v, g in zip(p, a)]
        return tuple(x + p + a)

    point = torch.utils.checkpoint.checkpoint
    a = point(lambda *y: tuple(_pm_force(list(y), box, N, m)), *x, use_reentrant=False)
    s = tuple(x + p) + tuple(a)
    for K1, D, K2 in zip(*factors):
        s = point(step, float(K1), float(D), float(K2), *s, use_reentrant=False)
    delta = _deposit(list(s[:3]), box, N, 1.0) / (n ** 3 / N ** 3) - 1.0
    loss = 0.5 * ((delta.reshape(-1) - target) ** 2).sum()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": noise.grad.cpu().numpy()}
