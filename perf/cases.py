"""The calls this framework is timed on, through its public entry points.

Each case is one thing that a program using the framework does over and over: a transform between
physical and spectral space, the nonlinear term, the wall boundary conditions with the pressure
projection, a line of diagnostics, time steps of a solver, a step of a batched ensemble.  Sizes are
nx, ny (periodic) and nzp, the physical points of the wall-bounded direction (+25 FC-Gram points,
d = 5), from the framework's own configurations: 32 to 96 for ensemble members, 64 x 64 x 65 for the
plain channel, 64 to 256 for served requests, 256 x 256 x 257 and 512 x 512 x 513 for the large ones.

Inputs are made on the GPU from the seed with plain torch (a program's initial-condition code) and
written into the framework's device fields.  ``exact`` is the same mathematics in torch at 64 bits.
"""
from __future__ import annotations

import ctypes
import math
import os
import random

import numpy as np
import torch

from specter_gb300 import api

C, D = 25, 5  # FC-Gram continuation points and matching points
TABLES = os.path.join(os.path.dirname(os.path.abspath(api.__file__)), "tables")
KINDS = {"hd": api.HD, "bouss": api.BOUSS, "rotbouss": api.ROTBOUSS}
OMEGA = (0.1, 0.0, 0.5)


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a small member's forward transform: the smallest call, a few launches long
        dict(name="r2c_fp64_32x32x33", kind="r2c", prec="fp64", nx=32, ny=32, nzp=33, Lz=2.0),
        # output of a physical field of a served-size run (checkpoints, plots)
        dict(name="c2r_fp64_128x128x129", kind="c2r", prec="fp64", nx=128, ny=128, nzp=129, Lz=2.0),
        # initial conditions of a 256^2 run on the FP32-bulk form
        dict(name="r2c_fp32_256x256x257", kind="r2c", prec="fp32", nx=256, ny=256, nzp=257, Lz=1.0),
        # gradre and advect called one by one, as the Fortran driver does, on an uneven grid
        dict(name="nonlinear_fp64_96x64x97", kind="nonlinear", prec="fp64", nx=96, ny=64, nzp=97, Lz=2.0),
        # boundary conditions and projection called one by one, on an uneven grid
        dict(name="project_fp64_128x96x129", kind="project", prec="fp64", nx=128, ny=96, nzp=129, Lz=1.0),
        # a line of balance.txt / helicity.txt / noslip_diagnostic.txt
        dict(name="diagnostics_fp64_128x128x129", kind="diagnostics", prec="fp64", nx=128, ny=128, nzp=129, Lz=2.0),
        # the plain channel configuration, ten RK2 steps a call
        dict(name="step_channel_fp64_64x64x65", kind="step", prec="fp64", solver="hd", nx=64, ny=64, nzp=65, Lz=2.0,
             ord=2, steps=10, dt=1e-4, nu=1e-3),
        # a served convection request in the plain form
        dict(name="step_rb_fp64_256x256x257", kind="step", prec="fp64", solver="bouss", nx=256, ny=256, nzp=257, Lz=1.0,
             ord=2, steps=1, dt=1e-5, nu=1e-4),
        # the large convection run in the plain form
        dict(name="step_rb_fp64_512x512x513", kind="step", prec="fp64", solver="bouss", nx=512, ny=512, nzp=513, Lz=1.0,
             ord=2, steps=1, dt=1e-5, nu=1e-4),
        # the channel configuration of the precision form (FP32 nonlinear term), RK4
        dict(name="step_channel_mixed_256x256x257", kind="step", prec="mixed", solver="hd", nx=256, ny=256, nzp=257,
             Lz=2.0, ord=4, steps=1, dt=2e-5, nu=2e-4),
        # the large convection run in the precision form: the benchmark's workload
        dict(name="step_rb_mixed_512x512x513", kind="step", prec="mixed", solver="bouss", nx=512, ny=512, nzp=513,
             Lz=1.0, ord=2, steps=1, dt=1e-5, nu=1e-4),
        # a batched ensemble of uneven channels on the FP32-bulk form
        dict(name="ensemble_fp32_12", kind="ensemble", prec="fp32", members=12, grids=7, ord=2, steps=1, dt=1e-4,
             nu=1e-3),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(rng, lo, hi):
    """An even size: a usual transform length three times of four, else any even number (its half may
    be prime)."""
    if rng.random() < 0.75:
        usual = [n for n in (16, 24, 32, 40, 48, 60, 64, 80, 96, 100, 112, 128, 160, 192, 240, 256, 320, 384, 480, 512)
                 if lo <= n <= hi]
        want = _log_int(rng, lo, hi)
        return min(usual, key=lambda n: abs(math.log(n / want)))
    return 2 * _log_int(rng, lo // 2, hi // 2)


def _nzp(rng, lo, hi):
    """Physical z points (odd: nzp + 25 is even): the configurations' sizes half of the time."""
    if rng.random() < 0.5:
        return rng.choice([n for n in (33, 65, 97, 129, 257, 513) if lo <= n <= hi])
    return min(hi, _log_int(rng, lo, hi) | 1)


def draw(rng: random.Random):
    kind = rng.choice(["r2c", "c2r", "nonlinear", "project", "diagnostics", "step", "step", "step", "ensemble"])
    if kind == "ensemble":
        return dict(kind="ensemble", prec="fp32", members=rng.randint(2, 12), grids=rng.randint(100, 10000), ord=2,
                    steps=rng.randint(1, 4), dt=1e-4, nu=math.exp(rng.uniform(math.log(2e-4), math.log(2e-3))))
    hi = 512 if kind in ("r2c", "c2r") else 256
    nx, ny, nzp = _even(rng, 32, hi), _even(rng, 32, hi), _nzp(rng, 33, 513 if hi == 512 else 257)
    case = dict(kind=kind, prec=rng.choice(["fp64", "fp64", "fp32"]), nx=nx, ny=ny, nzp=nzp, Lz=rng.choice([1.0, 2.0]))
    if kind != "step":
        return case
    solver = rng.choice(["hd", "bouss", "bouss", "rotbouss"])
    case.update(prec=rng.choice(["fp64", "fp64", "mixed"]), solver=solver, ord=rng.choice([2, 2, 3, 4]),
                steps=rng.choice([1, 1, 2, 5]), dt=rng.choice([1e-5, 2e-5, 1e-4]),
                nu=math.exp(rng.uniform(math.log(1e-4), math.log(2e-3))))
    while case["nx"] * case["ny"] * (nzp + C) * case["ord"] * case["steps"] > 8e7:  # below the large plain run's cost
        if case["steps"] > 1:
            case["steps"] = 1
        elif case["nx"] >= case["ny"]:
            case["nx"] = case["nx"] // 4 * 2
        else:
            case["ny"] = case["ny"] // 4 * 2
    return case


def _members(case):
    """Grids of an ensemble: nx, ny and nzp of the ensemble configuration."""
    r = random.Random(case["grids"])
    return [dict(nx=r.choice((32, 48, 64, 96)), ny=r.choice((32, 48, 64, 96)), nzp=r.choice((33, 65, 97)), Lz=2.0)
            for _ in range(case["members"])]


# ------------------------------------------------------------------ the mathematics in torch, 64 bits
class Grid:
    """Wavenumbers, continuation matrix and transforms of one grid; complex fields are (nz, ny, nx/2+1)."""

    def __init__(self, c):
        self.nx, self.ny, self.nzp, self.Lz = c["nx"], c["ny"], c["nzp"], c["Lz"]
        self.nz = self.nzp + C
        dev = torch.device("cuda")
        A = np.fromfile(os.path.join(TABLES, f"A{C}-{D}.dat"), "f8").reshape(D, C).T
        Q = np.fromfile(os.path.join(TABLES, f"Q{D}.dat"), "f8").reshape(D, D).T
        W = A @ Q.T
        # continuation rows from the last D rows and (mirrored) the first D rows
        self.top = torch.tensor(W, device=dev, dtype=torch.complex128)
        self.bot = torch.tensor(np.ascontiguousarray(W[::-1, ::-1]), device=dev, dtype=torch.complex128)
        dz = self.Lz / (self.nzp - 1)
        self.z = dz * torch.arange(self.nz, device=dev, dtype=torch.float64)

        def freq(n, scale):
            k = torch.arange(n, device=dev, dtype=torch.float64)
            return torch.where(k < n // 2, k, k - n) * scale

        self.kx = freq(self.nx, 1.0)[: self.nx // 2 + 1].reshape(1, 1, -1)
        self.ky = freq(self.ny, 1.0).reshape(1, -1, 1)
        self.kz = freq(self.nz, 2 * math.pi / (dz * self.nz)).reshape(-1, 1, 1)
        self.k = (self.kx, self.ky, self.kz)

        def filt(k, n, scale):
            return torch.exp(-16 * math.log(10.0) * (2 * k / n / scale).pow(100))

        self.fc = (filt(self.kx, self.nx, 1.0) * filt(self.ky, self.ny, 1.0)
                   * filt(self.kz, self.nz, 2 * math.pi / (dz * self.nz)))
        self.k2 = self.kx ** 2 + self.ky ** 2 + self.kz ** 2
        self.kh = torch.sqrt(self.kx ** 2 + self.ky ** 2)[0]
        self.norm = float(self.nx) * self.ny * self.nz

    def fwd_z(self, f):
        """Mixed domain (physical rows) to spectral, with the continuation."""
        f = f[: self.nzp]
        ext = torch.einsum("ij,jyx->iyx", self.top, f[-D:]) + torch.einsum("ij,jyx->iyx", self.bot, f[:D])
        return torch.fft.fft(torch.cat([f, ext]), dim=0)

    def inv_z(self, f):
        return torch.fft.ifft(f, dim=0, norm="forward")

    def r2c(self, r):
        return self.fwd_z(torch.fft.rfft2(r[: self.nzp]))

    def c2r(self, f):
        g = torch.fft.ifft(self.inv_z(f), dim=1, norm="forward")
        return torch.fft.irfft(g, n=self.nx, dim=2, norm="forward")

    def deriv(self, f, d):
        return 1j * self.k[d] * f

    def advect(self, v, f):
        """(v . grad) f of spectral fields."""
        s = 0
        for d in range(3):
            s = s + self.c2r(v[d])[: self.nzp] * self.c2r(self.deriv(f, d))[: self.nzp]
        return self.r2c(s / self.norm ** 2)

    def project(self, v):
        """Pressure projection with zero normal velocity at the walls; returns (v, pr on physical rows)."""
        s = self.kx * v[0] + self.ky * v[1] + self.kz * v[2]
        k2 = self.k2.clone()
        k2[0, 0, 0] = 1.0
        d = -1j * s / k2
        d[0, 0, 0] = 0.0
        v = [v[i] - self.deriv(d, i) for i in range(3)]
        w = self.inv_z(v[2]) / self.nz
        b1, b2 = w[0], w[self.nzp - 1]
        kh = self.kh.clone()
        kh[0, 0] = 1.0
        e = torch.exp(-kh * self.Lz)
        t = 1.0 / (kh * (1 - torch.exp(-2 * kh * self.Lz)))
        c1, c2 = (b2 - b1 * e) * t, (-b1 + b2 * e) * t
        z = self.z[: self.nzp].reshape(-1, 1, 1)
        e1, e2 = torch.exp(kh * (z - self.Lz)), torch.exp(-kh * z)
        a, b = c1 * e1 + c2 * e2, kh * (c1 * e1 - c2 * e2)
        a[:, 0, 0] = b1[0, 0].real * z[:, 0, 0]
        b[:, 0, 0] = b1[0, 0].real
        pr = self.inv_z(d)[: self.nzp] / self.nz + a
        a, b = self.fwd_z(a), self.fwd_z(b)
        return [v[0] - self.deriv(a, 0), v[1] - self.deriv(a, 1), v[2] - b], pr

    def velocity_walls(self, v, pr, tmp):
        """No-slip walls corrected by the previous stage's pressure, then the projection."""
        for i in range(2):
            m = self.inv_z(v[i])[: self.nzp] / self.nz
            for w in (0, self.nzp - 1):
                m[w] = 0.0 if pr is None else self.deriv(pr[w : w + 1], i)[0] * tmp
                m[w, 0, 0] = 0.0
            v[i] = self.fwd_z(m)
        return self.project(v)

    def scalar_walls(self, th):
        m = self.inv_z(th)[: self.nzp] / self.nz
        m[0] = 0.0
        m[self.nzp - 1] = 0.0
        return self.fwd_z(m)

    def stage(self, c, o, v, th, pr, v0, th0):
        bouss, rot = c["solver"] != "hd", c["solver"] == "rotbouss"
        nl = [self.advect(v, f) for f in (v + [th] if bouss else v)]
        if rot:
            ox, oy, oz = OMEGA
            nl[0] = nl[0] + 2 * (oy * v[2] - oz * v[1])
            nl[1] = nl[1] + 2 * (oz * v[0] - ox * v[2])
            nl[2] = nl[2] + 2 * (ox * v[1] - oy * v[0])
        if bouss:
            nl[2] = nl[2] - th
            nl[3] = nl[3] - v[2]
        new = [old + c["dt"] / o * (-c["nu"] * self.k2 * f - self.fc * n)
               for old, f, n in zip(v0 + ([th0] if bouss else []), v + ([th] if bouss else []), nl)]
        tmp = 1 / o if o == c["ord"] else (o + 1) / o
        v, pr = self.velocity_walls(new[:3], pr, tmp)
        if bouss:
            th = self.scalar_walls(new[3])
            if not rot:
                th = self.r2c(self.c2r(th * self.fc) / self.norm)
        return v, th, pr

    def steps(self, c, v, th):
        pr = None
        for _ in range(c["steps"]):
            v0, th0 = v, th
            for o in range(c["ord"], 0, -1):
                v, th, pr = self.stage(c, o, list(v), th, pr, list(v0), th0)
        return v, th, pr

    # ---- initial conditions
    def _smooth(self, g, kmax):
        """Mixed-domain smooth random field a(z) and its z derivative: random x, y modes up to kmax times
        a few cosines in z."""
        modes = 6
        noise = torch.randn(modes, self.ny, self.nx, generator=g, device="cuda", dtype=torch.float64)
        spec = torch.fft.rfft2(noise) * ((self.kx ** 2 + self.ky ** 2) <= kmax ** 2)
        m = torch.arange(1, modes + 1, device="cuda", dtype=torch.float64).reshape(1, -1) * math.pi / self.Lz
        psi = 2 * math.pi * torch.rand(1, modes, generator=g, device="cuda", dtype=torch.float64)
        arg = m * self.z[: self.nzp].reshape(-1, 1) + psi
        f = torch.einsum("zm,myx->zyx", torch.cos(arg).to(spec.dtype), spec)
        return f, torch.einsum("zm,myx->zyx", (-m * torch.sin(arg)).to(spec.dtype), spec)

    def velocity(self, seed, amp=0.1):
        """Spectral Poiseuille flow plus a solenoidal perturbation that vanishes at the walls."""
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        kmax = max(2, min(32, self.nx // 4, self.ny // 4))
        z = self.z[: self.nzp].reshape(-1, 1, 1)
        env, denv = z ** 2 * (self.Lz - z) ** 2, 2 * z * (self.Lz - z) ** 2 - 2 * z ** 2 * (self.Lz - z)
        (a1, d1), (a2, d2), (a3, _) = (self._smooth(g, kmax) for _ in range(3))
        dx, dy = 1j * self.kx, 1j * self.ky
        u = [env * (dy * a3 - d2) - denv * a2, env * (d1 - dx * a3) + denv * a1, env * (dx * a2 - dy * a1)]
        rms = math.sqrt(sum(float((f.real ** 2 + f.imag ** 2).sum()) for f in u) * 2 / self.nzp) / (self.nx * self.ny)
        u = [f * (amp / rms) for f in u]
        u[0][:, 0, 0] += ((1 - (2 * z / self.Lz - 1) ** 2) * self.nx * self.ny).reshape(-1)
        return [self.fwd_z(f) for f in u]

    def theta(self, seed, amp=1e-3):
        """Spectral white noise between the walls."""
        g = torch.Generator(device="cuda").manual_seed(int(seed) + 7919)
        xi = torch.rand(self.nzp, self.ny, self.nx, generator=g, device="cuda", dtype=torch.float64) * 2 - 1
        z = self.z[: self.nzp].reshape(-1, 1, 1)
        return self.r2c(amp * xi * z * (self.Lz - z))

    def general(self, seed, count):
        """Spectral smooth random fields that vanish nowhere in particular (not solenoidal, wall values
        not zero)."""
        g = torch.Generator(device="cuda").manual_seed(int(seed) + 104729)
        return [self.fwd_z(self._smooth(g, max(2, min(16, self.nx // 4, self.ny // 4)))[0]) for _ in range(count)]

    def physical(self, seed):
        """A physical field on all nz rows: smooth plus noise."""
        g = torch.Generator(device="cuda").manual_seed(int(seed) + 15485863)
        f = torch.fft.irfft2(self._smooth(g, max(2, min(16, self.nx // 4, self.ny // 4)))[0], s=(self.ny, self.nx))
        r = torch.zeros(self.nz, self.ny, self.nx, device="cuda", dtype=torch.float64)
        r[: self.nzp] = f + 1e-3 * torch.randn(f.shape, generator=g, device="cuda", dtype=torch.float64)
        return r


# ------------------------------------------------------------------ device fields as tensors
class _Memory:
    """Device memory of `owner`, which lives as long as a tensor on it does."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=3, strides=None)


def view(field, solver=None):
    """The device memory of a field as a tensor: (nz, ny, nx/2+1) complex or (nz, ny, nx) real.  `solver`
    is the owner of a solver's own field."""
    p = field.plan
    ptr, nbytes = ctypes.c_void_p(), ctypes.c_longlong()
    api.check(p._L.specter_field_device_ptr(field.h, ctypes.byref(ptr), ctypes.byref(nbytes)))
    t = "<f8" if p.precision == api.FP64 else "<f4"
    if field.kind == api.REAL:
        return torch.as_tensor(_Memory((field, solver), ptr.value, (p.nz, p.ny, p.nx), t), device="cuda")
    flat = torch.as_tensor(_Memory((field, solver), ptr.value, (p.nz, p.ny, p.ldx, 2), t), device="cuda")
    return torch.view_as_complex(flat)[:, :, : p.nxh]


def _plan(c, prec):
    return api.Plan((c["nx"], c["ny"], c["nzp"] + C), (0, 0, C), (0, 0, D), (1.0, 1.0, c["Lz"]),
                    precision=api.FP32 if prec == "fp32" else api.FP64)


def _cdtype(c):
    return torch.complex64 if c["prec"] == "fp32" else torch.complex128


def _inputs(c, seed):
    """The arrays a case starts from, in the plan's precision."""
    g, kind = Grid(c), c["kind"]
    if kind == "r2c":
        return g, [g.physical(seed).to(torch.float32 if c["prec"] == "fp32" else torch.float64)]
    if kind == "c2r":
        arrays = [g.general(seed, 1)[0]]
    elif kind == "diagnostics":
        arrays = g.general(seed, 3)
    elif kind == "project":  # a velocity that is not yet solenoidal, and a scalar
        arrays = [a + 0.05 * b for a, b in zip(g.velocity(seed), g.general(seed, 3))] + [g.theta(seed)]
    else:
        arrays = g.velocity(seed)
        if kind == "nonlinear" or c.get("solver", "hd") != "hd":
            arrays.append(g.theta(seed))
    return g, [a.to(_cdtype(c)) for a in arrays]


def _fill(plan, fields, arrays):
    plan.synchronize()  # new fields are zeroed on the plan's stream
    for f, a in zip(fields, arrays):
        view(f).copy_(a)
    torch.cuda.synchronize()


# ------------------------------------------------------------------ prepare and run
def _prepare_solver(c, seed):
    plan = _plan(c, c["prec"])
    s = api.Solver(plan, KINDS[c["solver"]], ord=c["ord"], dt=c["dt"], nu=c["nu"], kappa=c["nu"], omega=OMEGA,
                   nl_fp32=c["prec"] == "mixed")
    _fill(plan, [f for f in (s.vx, s.vy, s.vz, s.th) if f is not None], _inputs(c, seed)[1])
    return dict(case=c, plan=plan, solver=s, state=[view(f, s) for f in s.state[:-1]], pr=view(s.pr, s)[: plan.nzp],
                stream=torch.cuda.ExternalStream(plan.stream))


def prepare(case, seed):
    if case["kind"] == "ensemble":
        members = [_prepare_solver(_member(case, m), seed * 1000 + i) for i, m in enumerate(_members(case))]
        return dict(case=case, members=members, batch=api.Batch([m["solver"] for m in members]))
    if case["kind"] == "step":
        return _prepare_solver(case, seed)
    plan = _plan(case, case["prec"])
    arrays = _inputs(case, seed)[1]
    kind = api.REAL if case["kind"] == "r2c" else api.COMPLEX
    f = [plan.field(kind) for _ in arrays]
    _fill(plan, f, arrays)
    st = dict(case=case, plan=plan, f=f)
    if case["kind"] == "r2c":
        st["out"] = [plan.field()]
    elif case["kind"] == "c2r":
        st["work"], st["out"] = plan.field(), [plan.field(api.REAL)]
    elif case["kind"] == "nonlinear":
        st["out"] = [plan.field() for _ in range(4)]
    elif case["kind"] == "project":
        st["pr"] = plan.field()
        st["out"] = f
    plan.synchronize()
    if "out" in st:
        st["views"] = [view(x) for x in st["out"]]
    if "pr" in st:
        st["views"].append(view(st["pr"])[: plan.nzp])
    return st


def _member(case, m):
    return dict(case, kind="step", solver="hd", **m)


def run(st):
    c = st["case"]
    kind = c["kind"]
    if kind == "ensemble":
        st["batch"].step(c["steps"])
        return [m["state"] + [m["pr"]] for m in st["members"]]
    p = st["plan"]
    if kind == "step":
        st["solver"].step(c["steps"])
        pr = st["pr"]
        if c["prec"] == "mixed":  # the precision form holds the pressure potential to FP32 accuracy: read as such
            with torch.cuda.stream(st["stream"]):
                pr = pr.to(torch.complex64)
        return st["state"] + [pr]
    f = st["f"]
    if kind == "r2c":
        api.fftp3d_real_to_complex(p, f[0], st["out"][0])
    elif kind == "c2r":  # the transform destroys its input
        st["work"].copy_from(f[0])
        api.fftp3d_complex_to_real(p, st["work"], st["out"][0])
    elif kind == "nonlinear":
        o = st["out"]
        api.gradre(p, f[0], f[1], f[2], o[0], o[1], o[2])
        api.advect(p, f[0], f[1], f[2], f[3], o[3])
    elif kind == "project":
        st["pr"].zero()
        api.v_imposebc_and_project(p, f[0], f[1], f[2], st["pr"], 1, 2)
        api.s_imposebc(p, f[3])
    else:
        bot, top = api.bouncheck_z(p, f[0], f[1])
        return [api.energy(p, f[0], f[1], f[2], 1), api.energy(p, f[0], f[1], f[2], 0),
                api.helicity(p, f[0], f[1], f[2]), api.divergence(p, f[0], f[1], f[2]), bot, top]
    return st["views"]


# ------------------------------------------------------------------ work and exact values
def work(case):
    """Inputs read once and outputs written once; transforms at 5 N log2 N a point (half of that for
    real data in x)."""
    if case["kind"] == "ensemble":
        w = [work(_member(case, m)) for m in _members(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    nx, ny, nzp = case["nx"], case["ny"], case["nzp"]
    nz, nxh = nzp + C, nx // 2 + 1
    real = 4.0 if case["prec"] == "fp32" else 8.0
    spec, mixed, phys = (2 * real * ny * nxh * nz, 2 * real * ny * nxh * nzp, real * nx * ny * nzp)
    fz, fxy = 5.0 * ny * nxh * nz * math.log2(nz), 2.5 * nx * ny * nzp * math.log2(nx * ny)
    kind = case["kind"]
    if kind == "r2c":
        return dict(bytes=phys + spec, flops=fz + fxy)
    if kind == "c2r":
        return dict(bytes=spec + phys * nz / nzp, flops=fz + fxy * nz / nzp)
    if kind == "nonlinear":  # v, theta and 9 + 3 derivatives back, 4 products forward
        return dict(bytes=8 * spec, flops=12 * fz + 20 * fxy)
    if kind == "project":  # three round trips in z, the wall values, the pressure, two profiles
        return dict(bytes=8 * spec + mixed, flops=9 * fz)
    if kind == "diagnostics":
        return dict(bytes=3 * spec, flops=7 * fz)
    nf = 3 if case["solver"] == "hd" else 4
    n = case["ord"] * case["steps"]
    return dict(bytes=case["steps"] * (2 * nf * spec + 2 * mixed), flops=n * ((2 * nf + nf + 9) * fz + 5 * nf * fxy))


def _exact_steps(case, seed):
    g, arrays = _inputs(case, seed)
    a = [x.to(torch.complex128) for x in arrays]
    v, th, pr = g.steps(case, a[:3], a[3] if len(a) > 3 else None)
    return v + ([th] if th is not None else []) + [pr]


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return [_exact_steps(_member(case, m), seed * 1000 + i) for i, m in enumerate(_members(case))]
    if kind == "step":
        return _exact_steps(case, seed)
    g, a = _inputs(case, seed)
    if kind == "r2c":
        return [g.r2c(a[0].double())]
    a = [x.to(torch.complex128) for x in a]
    if kind == "c2r":
        return [g.c2r(a[0])]
    if kind == "nonlinear":
        return [g.advect(a[:3], f) for f in a]
    if kind == "project":
        v, pr = g.velocity_walls(a[:3], None, 0.0)
        return v + [g.scalar_walls(a[3]), pr]
    weight = torch.full((1, 1, g.nx // 2 + 1), 2.0, device="cuda", dtype=torch.float64)
    weight[..., 0] = 1.0
    curl = [g.deriv(a[2], 1) - g.deriv(a[1], 2), g.deriv(a[0], 2) - g.deriv(a[2], 0), g.deriv(a[1], 0) - g.deriv(a[0], 1)]

    def mean(x, y):
        p = (g.inv_z(x) * g.inv_z(y).conj()).real[: g.nzp]
        return float((p * weight).sum()) / g.norm ** 2 / g.nzp

    div = sum(g.deriv(a[i], i) for i in range(3))
    walls = [sum(float(((g.inv_z(a[i])[w].abs() ** 2) * weight[0]).sum()) for i in range(2)) / g.norm ** 2
             for w in (0, g.nzp - 1)]
    return [sum(mean(f, f) for f in a), mean(curl[0], curl[0]) + 2 * mean(curl[1], curl[1]),
            sum(mean(a[i], curl[i]) for i in range(3)), mean(div, div)] + walls
