"""The work that a user of vonkarman_gb300 has it do, as measurable cases.

Three kinds of pass, each through the public entry points:

* ``step`` -- ``Periodic3D.run`` / ``step`` over some time steps, as a simulation's
  output interval: Tier-1 records and E(k) where asked for, then the new state
  handed to the caller (in page-locked buffers; single precision runs hand it on as
  complex64 on the GPU).
* ``grad`` -- one gradient of the final enstrophy by ``adjoint_forward`` and
  ``adjoint_backward``.
* ``fft``  -- a round trip of the ``FftBackend`` on device arrays: forward, a copy
  of the spectrum (the inverse overwrites its input), inverse.

Grids are the ones the solver accepts (cubic powers of two, 8..512); the FFT
backend takes any mix of 2^a and 3 * 2^a lengths.
"""

import ctypes
import math

import numpy as np
import torch
import torch.utils.checkpoint

from vonkarman_gb300 import GpuFftBackend, GridSpec, Periodic3D, SolverOptions, energy_spectrum
from vonkarman_gb300 import _native as nat

TWO_PI = 2.0 * math.pi
TIER1 = ("time", "dt", "energy", "enstrophy", "helicity", "superhelicity", "max_vorticity",
         "energy_dissipation_rate", "helicity_dissipation_rate", "cfl_number")


def _step(name, n, precision, steps, ic, *, every=0, spectrum=False, etd="reference", integrator="etd-rk4",
          dt=0.0, l=TWO_PI, nu=1e-3):
    return {"name": name, "kind": "step", "n": n, "precision": precision, "steps": steps, "ic": ic, "every": every,
            "spectrum": spectrum, "etd": etd, "integrator": integrator, "dt": dt, "l": l, "nu": nu}


def _grad(name, n, precision, steps, nsnap, schedule, *, dt=2e-3, nu=1e-2):
    return {"name": name, "kind": "grad", "n": n, "precision": precision, "steps": steps, "nsnap": nsnap,
            "schedule": schedule, "dt": dt, "nu": nu}


def _fft(name, nx, ny, nz, precision):
    return {"name": name, "kind": "fft", "nx": nx, "ny": ny, "nz": nz, "precision": precision}


def listed():
    return [
        # a small grid stepped with a record every step (parameter sweeps, CI runs): launches and latency
        _step("step_n16_fp64", 16, "fp64", 1, "iso", every=1),
        # the Taylor-Green validation run: Tier-1 after every step
        _step("step_tg_n64_fp64", 64, "fp64", 10, "tg", every=1, nu=1.0 / 1600.0),
        # classical RK4 with a fixed dt, the integrator the ETD scheme is checked against
        _step("step_rk4_n128_fp64", 128, "fp64", 2, "abc", integrator="rk4", dt=2e-3, nu=1e-2),
        # exploratory turbulence in single precision, E(k) and Tier-1 at the output interval
        _step("step_n128_fp32", 128, "fp32bulk", 20, "iso", every=10, spectrum=True),
        # the benchmark's workload: random isotropic turbulence, adaptive CFL, E(k)
        _step("step_n256_fp64", 256, "fp64", 2, "iso", spectrum=True),
        _step("step_n256_fp32", 256, "fp32bulk", 10, "iso", spectrum=True),
        # the large workload: anti-parallel vortex tubes
        _step("step_tubes_n512_fp32", 512, "fp32bulk", 4, "tubes"),
        # a gradient for optimal-perturbation ascent (two-level checkpoints), double precision
        _grad("grad_n128_fp64", 128, "fp64", 4, 2, "two-level"),
        # the same in single precision with the memory-saving schedule
        _grad("grad_n256_fp32", 256, "fp32bulk", 6, 3, "binomial", dt=1e-3, nu=2e-3),
        # the FFT backend alone: an anisotropic grid in double, a large cube in single precision
        _fft("fft_192x256x384_fp64", 192, 256, 384, "fp64"),
        _fft("fft_512x512x512_fp32", 512, 512, 512, "fp32bulk"),
        # a small transform called on its own
        _fft("fft_24x32x48_fp64", 24, 32, 48, "fp64"),
    ]


def draw(rng):
    kind = rng.choice(("step", "step", "step", "grad", "fft"))
    precision = rng.choice(("fp64", "fp32bulk"))
    if kind == "fft":
        lens = (8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512)
        c = _fft("", rng.choice(lens), rng.choice(lens), rng.choice(lens), precision)
    elif kind == "grad":
        n = rng.choice((16, 32, 64, 128))
        steps = rng.randint(2, 5)
        c = _grad("", n, precision, steps, rng.randint(2, steps), rng.choice(("two-level", "binomial")),
                  dt=rng.uniform(5e-4, 2e-3), nu=10.0 ** rng.uniform(-3.0, -2.0))
    else:
        n = rng.choice((8, 16, 32, 64, 128, 256))
        steps = rng.randint(1, 2 if n == 256 and precision == "fp64" else 9)
        integrator = rng.choice(("etd-rk4", "etd-rk4", "rk4"))
        c = _step("", n, precision, steps, rng.choice(("iso", "abc", "tg", "tubes")), every=rng.choice((0, 1, 2)),
                  spectrum=rng.choice((False, True)), etd=rng.choice(("reference", "cox-matthews")),
                  integrator=integrator, dt=rng.choice((0.0, 5e-4)), l=rng.choice((TWO_PI, rng.uniform(3.0, 9.0))),
                  nu=10.0 ** rng.uniform(-3.5, -2.0))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# initial states (torch, on the GPU)
# ---------------------------------------------------------------------------
def _wave(n, l):
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    k = torch.where(k < n // 2, k, k - n) * (TWO_PI / l)
    kz = torch.arange(n // 2 + 1, dtype=torch.float64, device="cuda") * (TWO_PI / l)
    return k[:, None, None], k[None, :, None], kz[None, None, :]


def _project(u, n, l):
    kx, ky, kz = _wave(n, l)
    k2 = kx * kx + ky * ky + kz * kz
    inv = torch.where(k2 > 0, 1.0 / torch.where(k2 > 0, k2, 1.0), 0.0)
    d = (kx * u[0] + ky * u[1] + kz * u[2]) * inv
    return [u[0] - kx * d, u[1] - ky * d, u[2] - kz * d]


def _energy(u, n):
    w = torch.full((n // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    w[0] = w[n // 2] = 1.0
    return 0.5 * sum(float((w * (c.real.square() + c.imag.square())).sum()) for c in u) / float(n) ** 6


def _turbulence(n, l, kp, energy, gen):
    """Random solenoidal field with E(k) ~ (k/kp)^4 / (1 + (k/kp)^2)^(17/6)."""
    kx, ky, kz = _wave(n, l)
    k = torch.sqrt(kx * kx + ky * ky + kz * kz)
    amp = torch.where(k > 0, (k / kp) / (1.0 + (k / kp) ** 2) ** (17.0 / 12.0), 0.0)
    u = []
    for _ in range(3):
        noise = torch.randn((n, n, n), dtype=torch.float64, device="cuda", generator=gen)
        u.append(torch.fft.rfftn(noise) * amp)
    u = _project(u, n, l)
    s = math.sqrt(energy / _energy(u, n))
    return [c * s for c in u]


def _initial(ic, n, l, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if ic == "iso":
        return _turbulence(n, l, 4.0 * TWO_PI / l, 0.5, gen)
    x = torch.arange(n, dtype=torch.float64, device="cuda") * (TWO_PI / n)
    X, Y, Z = x[:, None, None], x[None, :, None], x[None, None, :]
    one = torch.ones((n, n, n), dtype=torch.float64, device="cuda")
    if ic == "tubes":
        # two z-aligned Gaussian vortex tubes, their distance and displacement seeded
        r = torch.rand(2, dtype=torch.float64, generator=torch.Generator().manual_seed(int(seed)))
        sep, eps, sigma = 0.9 + 0.2 * float(r[0]), 0.08 + 0.04 * float(r[1]), 0.35
        wz = torch.zeros((n, n, n), dtype=torch.float64, device="cuda")
        for sign, yc in ((1.0, math.pi - 0.5 * sep), (-1.0, math.pi + 0.5 * sep)):
            dx = X - (math.pi + eps * torch.sin(Z))
            wz += sign / (math.pi * sigma * sigma) * torch.exp(-(dx * dx + (Y - yc) ** 2) / (sigma * sigma))
        w = torch.fft.rfftn(wz)
        kx, ky, kz = _wave(n, TWO_PI)
        k2 = kx * kx + ky * ky + kz * kz
        w = w * torch.where(k2 > 0, 1.0 / torch.where(k2 > 0, k2, 1.0), 0.0)
        return _project([1j * ky * w, -1j * kx * w, torch.zeros_like(w)], n, TWO_PI)
    if ic == "tg":
        u = [torch.sin(X) * torch.cos(Y) * torch.cos(Z), -torch.cos(X) * torch.sin(Y) * torch.cos(Z), 0.0 * one]
    else:   # abc
        u = [(torch.sin(Z) + torch.cos(Y)) * one, (torch.sin(X) + torch.cos(Z)) * one,
             (torch.sin(Y) + torch.cos(X)) * one]
    pert = _turbulence(n, l, 8.0 * TWO_PI / l, 0.5e-4, gen)   # rms 1e-2
    return [torch.fft.rfftn(c) + p for c, p in zip(u, pert)]


# ---------------------------------------------------------------------------
# what a program keeps
# ---------------------------------------------------------------------------
class _Solver:
    def __init__(self, case, u, options):
        self.solver = Periodic3D(GridSpec(case["n"], case.get("l", TWO_PI)), case["nu"],
                                 [c.cpu().numpy() for c in u], options)
        shape = self.solver.grid.spectral_shape
        self.buf = [torch.empty(shape, dtype=torch.complex128, pin_memory=True).numpy() for _ in range(3)]

    def state(self):
        s = self.solver
        nat.check(s._lib.vk_get_state_host(s._ctx, *[nat.dptr(a) for a in self.buf]), s._lib, s._ctx)
        return self.buf


class _Fft:
    def __init__(self, case, x):
        dims = (case["nx"], case["ny"], case["nz"])
        self.plan = GpuFftBackend(*dims, precision=case["precision"])
        self.stream = torch.cuda.Stream()
        cdt = torch.complex64 if case["precision"] == "fp32bulk" else torch.complex128
        half = (dims[0], dims[1], dims[2] // 2 + 1)
        self.x = x
        self.X = torch.empty(half, dtype=cdt, device="cuda")
        self.W = torch.empty_like(self.X)
        self.y = torch.empty_like(x)


def _options(case):
    return SolverOptions(precision=case["precision"], etd_variant=case["etd"], integrator=case["integrator"],
                         dt_mode="fixed" if case["dt"] else "cfl", dt_fixed=case["dt"])


def _field(case, seed):
    dt = torch.float32 if case["precision"] == "fp32bulk" else torch.float64
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.randn((case["nx"], case["ny"], case["nz"]), dtype=torch.float64, device="cuda", generator=gen)
    return x.to(dt)


def prepare(case, seed):
    if case["kind"] == "fft":
        s = _Fft(case, _field(case, seed))
    elif case["kind"] == "grad":
        opts = SolverOptions(precision=case["precision"], dt_mode="fixed", dt_fixed=case["dt"])
        s = _Solver(case, _initial("abc", case["n"], TWO_PI, seed), opts)
    else:
        s = _Solver(case, _initial(case["ic"], case["n"], case["l"], seed), _options(case))
    torch.cuda.synchronize()
    return {"case": case, "work": s}


def run(state):
    case, s = state["case"], state["work"]
    single = case["precision"] == "fp32bulk"
    if case["kind"] == "fft":
        lib, h, st = s.plan._lib, s.plan._h, ctypes.c_void_p(s.stream.cuda_stream)
        nat.check(lib.vk_fft_r2c_device(h, ctypes.c_void_p(s.x.data_ptr()), ctypes.c_void_p(s.X.data_ptr()), st),
                  lib, fft=h)
        with torch.cuda.stream(s.stream):
            s.W.copy_(s.X)
        nat.check(lib.vk_fft_c2r_device(h, ctypes.c_void_p(s.W.data_ptr()), ctypes.c_void_p(s.y.data_ptr()), st),
                  lib, fft=h)
        return {"X": s.X, "y": s.y}
    if case["kind"] == "grad":
        value = s.solver.adjoint_forward(case["steps"], case["nsnap"], case["schedule"])
        g = s.solver.adjoint_backward()
        if single:   # handed on in the precision it was computed in
            return {"J": value, "g": [torch.from_numpy(c).cuda().to(torch.complex64) for c in g]}
        return {"J": np.float64(value), "g": g}
    out = {}
    if case["every"]:
        rec = s.solver.run(case["steps"], case["every"])
        t1 = np.array([[getattr(r, f) for f in TIER1] for r in rec])
        out["tier1"] = t1.astype(np.float32) if single else t1
    else:
        s.solver.step(case["steps"])
    if case["spectrum"]:
        e = energy_spectrum(s.solver)[1]
        out["spectrum"] = e.astype(np.float32) if single else e
    u = s.state()
    out["u"] = [torch.from_numpy(c).cuda().to(torch.complex64) for c in u] if single else u
    return out


# ---------------------------------------------------------------------------
# necessary work
# ---------------------------------------------------------------------------
def _fft_flops(points):
    """One real transform of `points` values."""
    return 2.5 * points * math.log2(points)


def work(case):
    c = 4 if case["precision"] == "fp32bulk" else 8
    if case["kind"] == "fft":
        pts = case["nx"] * case["ny"] * case["nz"]
        half = case["nx"] * case["ny"] * (case["nz"] // 2 + 1)
        return {"bytes": c * (2 * pts + 2 * 2 * half), "flops": 2 * _fft_flops(pts)}
    n = case["n"]
    m3, n3, modes = (3 * n // 2) ** 3, n ** 3, n * n * (n // 2 + 1)
    nonlinear = 9 * _fft_flops(m3) + 9 * m3 + 20 * modes
    state = 3 * modes * 2 * c
    if case["kind"] == "grad":
        # forward, the stages rebuilt, the transposed evaluations (15 transforms)
        adjoint = 15 * _fft_flops(m3) + 18 * m3 + 40 * modes
        return {"bytes": 2 * state, "flops": case["steps"] * 4 * (2 * nonlinear + adjoint)}
    flops = case["steps"] * (4 * nonlinear + (0 if case["dt"] else 3 * _fft_flops(n3)))
    return {"bytes": 2 * state, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits by plain torch
# ---------------------------------------------------------------------------
def _c2r(xh, m):
    return torch.fft.irfft(torch.fft.ifftn(xh, dim=(0, 1)), n=m, dim=2)


class _Plain:
    def __init__(self, n, l, nu):
        self.n, self.m, self.nu = n, 3 * n // 2, nu
        self.l = l
        self.kx, self.ky, self.kz = _wave(n, l)
        self.k2 = self.kx * self.kx + self.ky * self.ky + self.kz * self.kz

    def curl(self, u):
        kx, ky, kz = self.kx, self.ky, self.kz
        return [1j * (ky * u[2] - kz * u[1]), 1j * (kz * u[0] - kx * u[2]), 1j * (kx * u[1] - ky * u[0])]

    def physical(self, c):
        n, m, h = self.n, self.m, self.n // 2
        lo = torch.cat((c[:h], c.new_zeros((m - n,) + tuple(c.shape[1:])), c[h:]), 0)
        p = torch.cat((lo[:, :h], lo.new_zeros((m, m - n, lo.shape[2])), lo[:, h:]), 1)
        p = torch.cat((p, p.new_zeros((m, m, m // 2 - h))), 2)
        return _c2r(p, m) * (float(m) / n) ** 3

    def spectral(self, f):
        n, m, h = self.n, self.m, self.n // 2
        g = torch.fft.rfftn(f)[:, :, :h + 1]
        g = torch.cat((g[:h], g[m - h:]), 0)
        return torch.cat((g[:, :h], g[:, m - h:]), 1) * (float(n) / m) ** 3

    def nonlinear(self, u):
        a = [self.physical(c) for c in u]
        w = [self.physical(c) for c in self.curl(u)]
        r = [self.spectral(a[(i + 1) % 3] * w[(i + 2) % 3] - a[(i + 2) % 3] * w[(i + 1) % 3]) for i in range(3)]
        return _project(r, self.n, self.l)

    def cfl(self, u):
        v = sum(_c2r(c, self.n).square() for c in u).max().sqrt().item()
        dx = self.l / self.n
        return 0.5 * min(min(dx / v if v > 1e-30 else 1.0, dx * dx / self.nu), 0.1)

    def table(self, dt):
        z = -self.nu * self.k2 * dt

        def phi(z):
            s1 = s2 = s3 = 0.0
            for j in range(32):
                th = TWO_PI * (j + 0.5) / 32
                w = z + complex(math.cos(th), math.sin(th))
                ew = torch.exp(w)
                s1 = s1 + ((ew - 1.0) / w).real
                s2 = s2 + ((ew - 1.0 - w) / (w * w)).real
                s3 = s3 + ((ew - 1.0 - w - 0.5 * w * w) / (w * w * w)).real
            return s1 / 32, s2 / 32, s3 / 32

        # phi depends on |k|^2 alone: tabulate the distinct values
        v, inv = torch.unique(z, return_inverse=True)
        f1, f2, f3 = phi(v)
        h1 = phi(0.5 * v)[0]
        return [t[inv] for t in (torch.exp(v), torch.exp(0.5 * v), h1, f1, f1 - 3 * f2 + 4 * f3, 2 * f2 - 4 * f3,
                                 4 * f3 - f2)]

    def etd_step(self, u, dt, tab, variant):
        full, half, a21, a41, b1, b23, b4 = tab
        q = dt * a21 if variant == "reference" else 0.5 * dt * a21
        n1 = self.nonlinear(u)
        a = [half * u[i] + q * n1[i] for i in range(3)]
        n2 = self.nonlinear(a)
        n3 = self.nonlinear([half * u[i] + q * n2[i] for i in range(3)])
        if variant == "reference":
            c = [full * u[i] + dt * a41 * (2.0 * n3[i] - n1[i]) for i in range(3)]
        else:
            c = [half * a[i] + q * (2.0 * n3[i] - n1[i]) for i in range(3)]
        n4 = self.nonlinear(c)
        return [full * u[i] + dt * (b1 * n1[i] + b23 * (n2[i] + n3[i]) + b4 * n4[i]) for i in range(3)]

    def rk4_step(self, u, dt):
        def rhs(s):
            r = self.nonlinear(s)
            return [r[i] - self.nu * self.k2 * s[i] for i in range(3)]

        k1 = rhs(u)
        k2 = rhs([u[i] + 0.5 * dt * k1[i] for i in range(3)])
        k3 = rhs([u[i] + 0.5 * dt * k2[i] for i in range(3)])
        k4 = rhs([u[i] + dt * k3[i] for i in range(3)])
        return [u[i] + dt / 6.0 * (k1[i] + 2.0 * k2[i] + 2.0 * k3[i] + k4[i]) for i in range(3)]

    def weight(self):
        w = torch.full((self.n // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
        w[0] = w[self.n // 2] = 1.0
        return w

    def dot(self, a, b):
        w = self.weight()
        return sum((w * (x.real * y.real + x.imag * y.imag)).sum() for x, y in zip(a, b)) / float(self.n) ** 6

    def tier1(self, u, time, dt):
        o = self.curl(u)
        ens, hel = self.dot(o, o).item(), self.dot(u, o).item()
        sup = self.dot(o, self.curl(o)).item()
        wm = sum(_c2r(c, self.n).square() for c in o).max().sqrt().item()
        return [time, dt, 0.5 * self.dot(u, u).item(), ens, hel, sup, wm, -2.0 * self.nu * ens, -2.0 * self.nu * sup,
                wm * dt / (self.l / self.n)]

    def spectrum(self, u):
        ns = int(math.ceil(math.sqrt(3.0) * (self.n // 2))) + 1
        shell = torch.floor(torch.sqrt(self.k2) + 0.5).long().reshape(-1)
        e = sum(c.real.square() + c.imag.square() for c in u)
        e = (0.5 * self.weight() * e / float(self.n) ** 6).reshape(-1)
        keep = shell < ns
        return torch.zeros(ns, dtype=torch.float64, device="cuda").index_add_(0, shell[keep], e[keep])


def exact(case, seed):
    if case["kind"] == "fft":
        x = _field(case, seed).double()
        return {"X": torch.fft.rfftn(x), "y": x}
    if case["n"] > 256 or case["n"] ** 3 * case["steps"] > 10 * 256 ** 3:
        return None
    if case["kind"] == "grad":
        if case["n"] > 128:
            return None
        p = _Plain(case["n"], TWO_PI, case["nu"])
        u0 = [c.requires_grad_() for c in _initial("abc", case["n"], TWO_PI, seed)]
        u, tab = u0, p.table(case["dt"])
        for _ in range(case["steps"]):
            u = torch.utils.checkpoint.checkpoint(
                lambda *a: tuple(p.etd_step(list(a), case["dt"], tab, "reference")), *u, use_reentrant=False)
        o = p.curl(list(u))
        value = p.dot(o, o)
        g = torch.autograd.grad(value, u0)
        # L2 inner product of the physical fields, real solenoidal Nyquist-free fields
        n = case["n"]
        g = [c * float(n) ** 6 / p.weight() for c in g]
        keep = torch.ones((n, n, n // 2 + 1), dtype=torch.float64, device="cuda")
        keep[n // 2], keep[:, n // 2], keep[:, :, n // 2] = 0.0, 0.0, 0.0
        g = _project([c * keep for c in g], n, TWO_PI)
        return {"J": value.item(), "g": [torch.fft.rfftn(_c2r(c, n)) for c in g]}
    p = _Plain(case["n"], case["l"], case["nu"])
    u = _initial(case["ic"], case["n"], case["l"], seed)
    dt = case["dt"] or p.cfl(u)
    etd = case["integrator"] == "etd-rk4"
    tab = p.table(dt) if etd else None
    time, rec = 0.0, []
    for i in range(case["steps"]):
        if not case["dt"]:
            new = p.cfl(u)
            if abs(new - dt) / max(dt, 1e-30) > 0.01:
                dt = new
                tab = p.table(dt) if etd else None
        u = p.etd_step(u, dt, tab, case["etd"]) if etd else p.rk4_step(u, dt)
        time += dt
        if case["every"] and (i + 1) % case["every"] == 0:
            rec.append(p.tier1(u, time, dt))
    out = {"u": u}
    if case["every"]:
        out["tier1"] = np.array(rec).reshape(len(rec), len(TIER1))
    if case["spectrum"]:
        out["spectrum"] = p.spectrum(u)
    return out
