"""Performance cases: what a user of this solver has it do.

A case is a dict of plain values.  Its ``kind`` says which public call it is:

``step``      one split step (``GpuOneStep`` of the reference), field in place
``march``     ``steps`` serial fine steps (``Solver.run``), field in place
``parareal``  one Parareal solve (``Solver.parareal``)
``batch``     several Parareal solves of mixed sizes at once (``batch_solve``)

and its ``vel`` the setting: ``const`` (vx, vy), ``rot`` (solid-body rotation)
and ``swirl`` (time-dependent deformation) are periodic on the unit square with
the time-consistent scheme; ``ref`` is the reference program's own setting
(domain [-1, 1]^2, velocity (-4y, 4x), its boundaries and its scheme).

``exact`` is a plain torch FP64 evaluation of the same scheme.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("parareal-cc-cfv-split-gpu_b200"))
import ccfv  # noqa: E402

DEV = "cuda"
OMEGA = 2.0 * math.pi


def listed():
    return [
        # the smallest call: one step of the reference program's own setting
        dict(name="step_ref_128", kind="step", vel="ref", nx=128, ny=128, K=1e-3),
        # a time loop on an odd, ragged grid that is not square
        dict(name="march_const_333x517", kind="march", vel="const", vx=1.0, vy=-0.7, nx=333,
             ny=517, K=1e-3, steps=10),
        # the reference program's serial fine loop at an ordinary and at a large size
        dict(name="march_ref_600", kind="march", vel="ref", nx=600, ny=600, K=1e-3, steps=10),
        dict(name="march_ref_2048", kind="march", vel="ref", nx=2048, ny=2048, K=1e-3, steps=8),
        # serial fine stepping of the benchmark's rotation
        dict(name="march_rot_2048", kind="march", vel="rot", nx=2048, ny=2048, K=1e-3, steps=8),
        # a caller that steps by itself on the largest benchmark grid
        dict(name="step_rot_4096", kind="step", vel="rot", nx=4096, ny=4096, K=1e-4),
        # strong diffusion (K dt / h^2 of about 20)
        dict(name="march_stiff_1024", kind="march", vel="const", vx=1.0, vy=1.0, nx=1024,
             ny=1024, K=0.05, steps=8),
        # feet that differ from cell to cell and with time
        dict(name="march_swirl_1024", kind="march", vel="swirl", nx=1024, ny=1024, K=1e-4,
             steps=6),
        # the small plain Parareal problem: 16 slices, one coarse step each
        dict(name="parareal_const_128", kind="parareal", vel="const", vx=1.0, vy=1.0, nx=128,
             ny=128, K=1e-2, nt=160, slices=16, ratio=10, prec=ccfv.FP64, T=1.0),
        # the rotation benchmark: one revolution, 64 slices, coarse dt = 8 x fine
        dict(name="parareal_rot_1024", kind="parareal", vel="rot", nx=1024, ny=1024, K=1e-3,
             nt=4096, slices=64, ratio=8, prec=ccfv.FP64, T=1.0),
        # the reference program's Parareal: 40 slices, standard form, 8 iterations
        dict(name="parareal_ref_256", kind="parareal", vel="ref", nx=256, ny=256, K=1e-3, nt=640,
             slices=40, ratio=0, prec=ccfv.FP64, T=1.0),
        # many problems at once, FP32 coarse steps
        dict(name="batch_12", kind="batch", count=12, nmin=64, nmax=640, T=1.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case of the same ranges."""
    what = rng.choice(["step", "march", "march", "march", "parareal", "batch"])
    if what == "batch":
        return dict(kind="batch", count=rng.randint(4, 12), nmin=64,
                    nmax=int(_log(rng, 200, 560)), T=rng.uniform(0.25, 1.0))
    if what == "parareal":
        n = int(_log(rng, 96, 512))
        if rng.random() < 0.3:  # the reference's schedule: 40 slices of J fine steps
            n = int(_log(rng, 96, 288))
            return dict(kind="parareal", vel="ref", nx=n, ny=n, K=_log(rng, 5e-4, 5e-3),
                        nt=40 * max(2, round(n / 16)), slices=40, ratio=0, prec=ccfv.FP64, T=1.0)
        slices, ratio = rng.choice([16, 32]), 8
        vx, vy, T = rng.uniform(-2, 2), rng.uniform(-2, 2), rng.uniform(0.25, 1.0)
        nt = math.ceil(T * n * max(abs(vx), abs(vy), 0.1) / 0.8 / (slices * ratio)) * slices * ratio
        return dict(kind="parareal", vel="const", vx=vx, vy=vy, nx=n, ny=n, K=_log(rng, 1e-4, 5e-2),
                    nt=nt, slices=slices, ratio=ratio, prec=rng.choice([ccfv.FP64, ccfv.FP32]), T=T)
    vel = rng.choice(["const", "rot", "swirl", "ref"])
    nx = int(_log(rng, 96, 4096))
    ny = nx if vel == "ref" or rng.random() < 0.4 else min(4096, max(96, int(nx * _log(rng, 0.5, 2))))
    case = dict(kind=what, vel=vel, nx=nx, ny=ny,
                K=_log(rng, 1e-4, 5e-2 if vel in ("const", "rot") else 3e-3))
    if vel == "const":
        case.update(vx=rng.uniform(-2, 2), vy=rng.uniform(-2, 2))
    if what == "march":
        case["steps"] = max(2, min(rng.randint(2, 24), int(1.2e8 / (nx * ny))))
    return case


# ---- the state of a user's program ------------------------------------------


def _grid(c):
    if c["vel"] == "ref":
        return ccfv.make_grid(c["nx"], c["ny"], K=c["K"])
    vel, vp = {"const": (ccfv.VEL_CONST, (c.get("vx", 0.0), c.get("vy", 0.0))),
               "rot": (ccfv.VEL_ROTATION, (OMEGA, 0.5, 0.5)),
               "swirl": (ccfv.VEL_SWIRL, (1.5,))}[c["vel"]]
    return ccfv.make_grid(c["nx"], c["ny"], bc=ccfv.BC_PERIODIC, velocity=vel, vel_params=vp,
                          K=c["K"], scheme=ccfv.SCHEME_CONSISTENT)


def _dt(c):
    """Fine step at CFL 0.8 (Parareal cases name their step count)."""
    if "nt" in c:
        return c["T"] / c["nt"]
    size = 2.0 if c["vel"] == "ref" else 1.0
    wx, wy = {"const": (abs(c.get("vx", 0.0)), abs(c.get("vy", 0.0))), "rot": (math.pi, math.pi),
              "swirl": (1.0, 1.0), "ref": (4.0, 4.0)}[c["vel"]]
    return 0.8 * min(size / c["nx"] / max(wx, 0.1), size / c["ny"] / max(wy, 0.1))


def _field(c, seed):
    """A few seeded Gaussian humps on a small background."""
    gen = torch.Generator().manual_seed(int(seed) * 1000003 + c["nx"] * 4099 + c["ny"])
    r = torch.rand(4, 4, generator=gen, dtype=torch.float64).tolist()
    lo, size = (-1.0, 2.0) if c["vel"] == "ref" else (0.0, 1.0)
    x = ((torch.arange(c["nx"], dtype=torch.float64, device=DEV) + 0.5) / c["nx"])[:, None]
    y = ((torch.arange(c["ny"], dtype=torch.float64, device=DEV) + 0.5) / c["ny"])[None, :]
    f = torch.full((c["nx"], c["ny"]), 0.0 if lo < 0 else 0.1, dtype=torch.float64, device=DEV)
    for a, b, s, m in r:
        den = 2.0 * (0.04 + 0.04 * s) ** 2
        dx, dy = x - (0.3 + 0.4 * a), y - (0.3 + 0.4 * b)
        if lo == 0.0:  # nearest periodic image
            dx, dy = dx - dx.round(), dy - dy.round()
        f += (0.5 + 0.5 * m) * torch.exp(-dx * dx / den) * torch.exp(-dy * dy / den)
    return f.contiguous()


def _instances(c):
    """The problems of a batch: sizes spread over [nmin, nmax], constant
    velocities, diffusivities from 1e-4 to 1e-1 (the same for every seed)."""
    gen = torch.Generator().manual_seed(c["count"] * 7919 + c["nmax"])
    out = []
    for i in range(c["count"]):
        r = torch.rand(4, generator=gen, dtype=torch.float64).tolist()
        n = int(round(c["nmin"] * (c["nmax"] / c["nmin"]) ** ((i + r[0]) / c["count"])))
        vx, vy = 4.0 * r[1] - 2.0, 4.0 * r[2] - 2.0
        slices, ratio = min(64, max(16, 16 * 2 ** round(math.log2(n / 64)))), 8
        nt = math.ceil(c["T"] * n * max(abs(vx), abs(vy), 0.1) / 0.8 / (slices * ratio)) * slices * ratio
        out.append(dict(vel="const", vx=vx, vy=vy, nx=n, ny=n, K=1e-4 * 1000.0 ** r[3], nt=nt,
                        slices=slices, ratio=ratio, prec=ccfv.FP32, T=c["T"]))
    return out


def _options(c):
    """Parareal options: the reference's schedule, or to an update of 1e-10."""
    if c["vel"] == "ref":
        return dict(t0=0.0, t1=c["T"], nt_fine=c["nt"], n_slices=c["slices"], kmax=8)
    return dict(t0=0.0, t1=c["T"], nt_fine=c["nt"], n_slices=c["slices"], coarse_ratio=c["ratio"],
                tol=1e-10, kmax=c["slices"], coarse_precision=c["prec"], form=ccfv.FORM_DELTA,
                coarse_theta=ccfv.COARSE_THETA_AUTO)


def prepare(case, seed):
    if case["kind"] == "batch":
        problems = []
        for i, c in enumerate(_instances(case)):
            C0 = _field(c, seed + 31 * i)
            problems.append(dict(grid=_grid(c), C0=C0, C_T=torch.empty_like(C0), **_options(c)))
        return dict(case=case, problems=problems)
    state = dict(case=case, solver=ccfv.Solver(_grid(case)), C=_field(case, seed), t=0.0,
                 dt=_dt(case))
    if case["kind"] == "parareal":
        state["out"] = torch.empty_like(state["C"])
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        ccfv.batch_solve(state["problems"])
        return [p["C_T"] for p in state["problems"]]
    s, C, dt = state["solver"], state["C"], state["dt"]
    if case["kind"] == "parareal":
        s.parareal(C, state["out"], **_options(case))
        return state["out"]
    if case["kind"] == "step":
        s.step(C, state["t"], dt)
        state["t"] += dt
    else:
        s.run(C, state["t"], dt, case["steps"])
        state["t"] += case["steps"] * dt
    return C


def work(case):
    """A step reads and writes its field once; 3 sweeps of an eight-tap stencil
    (or per-cell feet, remap and derivative) and two recurrences per cell.  A
    Parareal solve cannot do less than one pass of its fine steps."""
    if case["kind"] == "batch":
        each = [work(dict(c, kind="parareal")) for c in _instances(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    n = {"step": 1, "march": case.get("steps"), "parareal": case.get("nt")}[case["kind"]]
    cells = float(case["nx"] * case["ny"]) * n
    return {"bytes": 16.0 * cells, "flops": (3 * 110.0 if case["vel"] == "swirl" else 60.0) * cells}


# ---- the scheme in plain torch FP64 -----------------------------------------


class _Scheme:
    """x(dt/2) y(dt) x(dt/2) split steps on fields [batch, nx, ny]."""

    def __init__(self, c, dt):
        self.c, self.dt = c, dt
        self.periodic = c["vel"] != "ref"
        self.lo, self.size = (0.0, 1.0) if self.periodic else (-1.0, 2.0)
        self.solve = {}  # (axis, Dt) -> LU factors of the line system

    def velocity(self, axis, s, tau, t):
        """Velocity along `axis` at position s along it, tau across it."""
        c, vel, sg = self.c, self.c["vel"], -1.0 if axis == 0 else 1.0
        if vel == "ref":
            return sg * 4.0 * tau + 0.0 * s
        if vel == "const":
            return c["vx" if axis == 0 else "vy"] + 0.0 * s + 0.0 * tau
        if vel == "rot":
            return sg * OMEGA * (tau - 0.5) + 0.0 * s
        w = torch.sin(math.pi * s) ** 2 * torch.sin(2.0 * math.pi * tau) * math.cos(math.pi * t / 1.5)
        return -sg * w

    def feet(self, axis, Dt, ta, tb):
        """Departure points of the edges, [L + 1, lines]: mean of the two Heun
        corner feet."""
        L, M = (self.c["nx"], self.c["ny"]) if axis == 0 else (self.c["ny"], self.c["nx"])
        s = (self.lo + self.size / L * torch.arange(L + 1, dtype=torch.float64, device=DEV))[:, None]
        tau = (self.lo + self.size / M * torch.arange(M + 1, dtype=torch.float64, device=DEV))[None, :]
        w0 = self.velocity(axis, s, tau, tb)
        f = s - 0.5 * Dt * (w0 + self.velocity(axis, s - Dt * w0, tau, ta))
        return 0.5 * (f[:, :-1] + f[:, 1:])

    def taps(self, c, k, derivative=False):
        """Cells k-2 .. k+2 of every line of c [batch, L, lines]."""
        L = c.shape[1]
        if self.periodic:
            rows = [torch.remainder(k + j, L) for j in range(-2, 3)]
            src = c
        else:  # two extrapolated ghost cells on either side
            a, b, d, p, q, r = c[:, 0], c[:, 1], c[:, 2], c[:, -1], c[:, -2], c[:, -3]
            g = [(-15 * d + 56 * b - 30 * a) / 11, (-d + 3 * b + 9 * a) / 11,
                 (-r + 3 * q + 9 * p) / 11, (-15 * r + 56 * q - 30 * p) / 11]
            src = torch.cat([torch.stack(g[:2], 1), c, torch.stack(g[2:], 1)], 1)
            rows = [k + j + 2 for j in range(-2, 3)]
            if derivative:  # the reference's choice of ghosts next to the ends
                rows[0] = torch.where(k == 1, 0, rows[0])
                rows[4] = torch.where(k == L - 2, L + 3, rows[4])
        return [src.gather(1, i[None].expand(c.shape[0], -1, -1)) for i in rows]

    def locate(self, f, h, L):
        k = torch.floor((f - self.lo) / h)
        if not self.periodic:
            k = k.clamp(0, L - 1)
        return k.long(), (f - (self.lo + h * k)) / h

    def integral(self, c, k, xi):
        """PPM integral of cell k from its left edge to xi."""
        m2, m1, z, p1, p2 = self.taps(c, k)
        cl = (7 * (z + m1) - (p1 + m2)) / 12
        cr = (7 * (p1 + z) - (p2 + m1)) / 12
        c6 = 6 * (z - 0.5 * (cl + cr))
        return -c6 * xi ** 3 / 3 + 0.5 * (cr - cl + c6) * xi ** 2 + cl * xi

    def remap(self, c, f, h, eps):
        L, fl, fr = c.shape[1], f[:-1], f[1:]
        if self.periodic:
            kl, xl = self.locate(fl, h, L)
            kr, xr = self.locate(fr, h, L)
        else:
            kl, xl = self.locate(fl.clamp(min=self.lo + eps), h, L)
            kr, xr = self.locate(fr.clamp(max=self.lo + self.size - eps), h, L)
        out = self.integral(c, kr, xr) - self.integral(c, kl, xl)
        for j in range(int((kr - kl).abs().max())):  # whole cells between the feet
            for near, far, sign in ((kl, kr, 1.0), (kr, kl, -1.0)):
                i = near + j
                rows = torch.remainder(i, L) if self.periodic else i.clamp(0, L - 1)
                x = c.gather(1, rows[None].expand(c.shape[0], -1, -1))
                out = out + torch.where(i < far, sign * x, 0.0)
        if not self.periodic:
            none = (fl > self.lo + self.size) | (fr < self.lo) | (fl == fr)
            out = torch.where(none, 0.0, out)
        return out

    def derivative(self, c, f, h):
        L = c.shape[1]
        g = f if self.periodic else f.clamp(self.lo + 1e-15, self.lo + self.size - 1e-15)
        k, x = self.locate(g, h, L)
        m2, m1, z, p1, p2 = self.taps(c, k, derivative=True)
        x2, x3 = x * x, x * x * x
        d = ((2 * x3 - 6 * x2 + 3 * x + 1) * m2 + (-8 * x3 + 18 * x2 + 6 * x - 15) * m1 +
             (12 * x3 - 18 * x2 - 24 * x + 15) * z + (-8 * x3 + 6 * x2 + 18 * x - 1) * p1 +
             (2 * x3 - 3 * x) * p2) / (12 * h)
        if not self.periodic:
            d = torch.where((f >= self.lo) & (f <= self.lo + self.size), d, 0.0)
        return d

    def sweep(self, c, axis, Dt, ta, tb, of_remap=False):
        """One sweep along dimension 1 of c [batch, L, lines]."""
        L = c.shape[1]
        h = self.size / L
        f = self.feet(axis, Dt, ta, tb)
        r = self.remap(c, f, h, 1e-15 if axis == 0 else 1e-16)
        d = self.derivative(r if of_remap else c, f, h)
        nu = self.c["K"] * Dt / (h * h)
        b = r + 0.5 * nu * h * (d[:, 1:] - d[:, :-1])
        pad = [b[:, -1:], b, b[:, :1]] if self.periodic else [0 * b[:, :1], b, 0 * b[:, :1]]
        e = torch.cat(pad, 1)
        m = (e[:, :-2] + 10 * b + e[:, 2:]) / 12
        if (axis, Dt) not in self.solve:
            off, eye = 1.0 / 12 - 0.5 * nu, torch.eye(L, dtype=torch.float64, device=DEV)
            A = (10.0 / 12 + nu) * eye + off * (eye.roll(1, 0) + eye.roll(-1, 0))
            if not self.periodic:
                A[0, -1] = A[-1, 0] = 0.0
            self.solve[axis, Dt] = torch.linalg.lu_factor(A)
        rhs = m.permute(1, 0, 2).reshape(L, -1)
        x = torch.linalg.lu_solve(*self.solve[axis, Dt], rhs)
        return x.reshape(L, c.shape[0], -1).permute(1, 0, 2)

    def step(self, c, t, dt=None):
        dt = self.dt if dt is None else dt
        c = self.sweep(c, 0, 0.5 * dt, t, t + 0.5 * dt)
        c = self.sweep(c.transpose(1, 2), 1, dt, t, t + dt).transpose(1, 2)
        return self.sweep(c, 0, 0.5 * dt, t + 0.5 * dt, t + dt, of_remap=not self.periodic)

    def spectra(self):
        """Uniform displacement on periodic lines: a sweep is a circular
        convolution of every line, here by the transform of its response to a
        single cell."""
        out = []
        for axis, Dt in ((0, 0.5 * self.dt), (1, self.dt)):
            L, M = (self.c["nx"], self.c["ny"]) if axis == 0 else (self.c["ny"], self.c["nx"])
            one = torch.zeros(1, L, M, dtype=torch.float64, device=DEV)
            one[:, 0] = 1.0
            out.append(torch.fft.rfft(self.sweep(one, axis, Dt, 0.0, Dt)[0], dim=0))
        return out

    def march(self, c, n):
        """n fine steps from t = 0 of a field [nx, ny]."""
        if n < 64 or self.c["vel"] not in ("const", "rot"):
            c = c[None]
            for k in range(n):
                c = self.step(c, k * self.dt)
            return c[0].contiguous()
        mx, my = self.spectra()
        nx, ny = c.shape
        if self.c["vel"] == "const":  # the same for every line: both directions at once
            full = torch.fft.fft(torch.fft.irfft(mx[:, 0], nx))
            m = full[:, None] ** 2 * my[None, :, 0]
            return torch.fft.irfft2(torch.fft.rfft2(c) * m ** n, (nx, ny))
        # the two half-sweeps between y-sweeps are one convolution
        c, my = torch.fft.irfft(torch.fft.rfft(c, dim=0) * mx, nx, dim=0), my.T.contiguous()
        for k in range(n):
            c = torch.fft.irfft(torch.fft.rfft(c, dim=1) * my, ny, dim=1)
            c = torch.fft.irfft(torch.fft.rfft(c, dim=0) * (mx if k == n - 1 else mx * mx), nx, dim=0)
        return c


def _exact_reference_parareal(c, C0):
    """The reference's schedule: one coarse step per slice, 8 iterations."""
    S, J, DT = c["slices"], c["nt"] // c["slices"], c["T"] / c["slices"]
    s = _Scheme(c, DT / J)
    U = [C0[None]]
    for _ in range(S):
        U.append(s.step(U[-1], 0.0, DT))
    G = list(U)
    for _ in range(8):
        F = []
        for part in torch.split(torch.cat(U[:S]), 8):
            for _ in range(J):  # the velocity does not depend on time
                part = s.step(part, 0.0)
            F += list(part.split(1))
        for n in range(S):
            g = s.step(U[n], 0.0, DT)
            U[n + 1], G[n + 1] = g + (F[n] - G[n + 1]), g
    return U[S][0].contiguous()


def exact(case, seed):
    if case["kind"] == "batch":
        return [exact(dict(c, kind="parareal"), seed + 31 * i) for i, c in enumerate(_instances(case))]
    if case["kind"] == "parareal":
        if case["vel"] == "ref":
            return _exact_reference_parareal(case, _field(case, seed))
        # converged to 1e-10: the serial fine solution
        return _Scheme(case, _dt(case)).march(_field(case, seed), case["nt"])
    return _Scheme(case, _dt(case)).march(_field(case, seed), case.get("steps", 1))
