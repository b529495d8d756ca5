"""The work that users of this library have it do, as cases to be timed and compared.

Every case is a dict of plain values; `kind` says which public entry points it goes through:

  stage        the two stages of an RK2 step on the caller's own device arrays (rk_stage_noalloc)
  run          `steps` time steps of a box (Solver.step), then the velocity (and scalar) state and the
               particles back on the host, as a driver does between two output steps
  particles    `steps` particle phases (Solver.particles_advance), then positions and velocities
  diagnostics  what a driver prints on an output step: shell spectra, one-dimensional spectra,
               velocity-gradient moments and the transfer spectrum
  ensemble     `steps` steps of independent boxes of uneven size, then every box's state

Initial fields are solenoidal with random phases and a model spectrum (k^4 at large scales, k^(-5/3) beyond
k = 3, an exponential tail), u' = 1; particles start at random positions.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "nasa-bluewater-psdns-benchmark-minsky_b200"))
import psdns_gpu as P  # noqa: E402

SIZES = (16, 32, 48, 64, 96, 128, 256, 512, 1024)
ENSEMBLE_SIZES = (32, 48, 64, 96)
# steps that an ensemble takes before it is measured: its sub-batches and tiles are chosen on real steps
ENSEMBLE_WARM = 32


def listed():
    def run(name, n, steps, prec="fp32", nc=0, rk=2, particles=0, forced=False, dt=0.0, kshift=1):
        return {"name": name, "kind": "run", "n": n, "steps": steps, "prec": prec, "nc": nc, "rk": rk,
                "particles": particles, "forced": forced, "dt": dt, "kshift": kshift}

    return [
        # the smallest call: a stage pair for a driver that owns its arrays
        {"name": "stage_32_fp32", "kind": "stage", "n": 32, "prec": "fp32"},
        # the plain 64^3 FP64 run with a fixed dt, 20 steps: launches and synchronisations count
        run("run_64_fp64", 64, 20, prec="fp64", dt=0.005),
        # a size that is no power of two, with a scalar
        run("run_96_scalar", 96, 20, nc=1, dt=0.003),
        # the shipped 128^3 input: RK4, kshift 4
        run("run_128_rk4", 128, 12, rk=4, dt=0.002, kshift=4),
        # 256^3 with a scalar and 2^16 particles, adaptive dt
        run("run_256_scalar_particles", 256, 20, nc=1, particles=65536),
        # the default 512^3 input, RK2
        run("run_512_fp32", 512, 12),
        # the same in FP64
        run("run_512_fp64", 512, 6, prec="fp64"),
        # the headline size, forced
        run("run_1024_forced", 1024, 8, forced=True),
        # many particles on one field: the interpolation and its spline coefficients
        {"name": "particles_512", "kind": "particles", "n": 512, "prec": "fp32", "particles": 1000001, "steps": 30},
        # an output step of a 512^3 run
        {"name": "diagnostics_512", "kind": "diagnostics", "n": 512, "prec": "fp32"},
        # a parameter sweep of small boxes
        {"name": "ensemble_32_boxes", "kind": "ensemble", "boxes": 32, "prec": "fp32", "steps": 160, "pick": 1},
    ]


def draw(rng):
    kind = rng.choice(("stage", "run", "run", "run", "run", "run", "particles", "diagnostics", "ensemble"))
    prec = rng.choice(("fp32", "fp32", "fp64"))
    if kind == "stage":
        return {"kind": kind, "n": rng.choice((16, 32, 64)), "prec": prec, "nu": round(0.004 * 4 ** rng.random(), 5)}
    if kind == "ensemble":
        return {"kind": kind, "boxes": rng.randint(5, 40), "prec": prec, "steps": rng.randint(20, 80),
                "pick": rng.randint(1, 1000)}
    if kind == "diagnostics":
        return {"kind": kind, "n": rng.choice((48, 64, 96, 128, 256, 512)), "prec": prec,
                "nu": round(0.001 * 4 ** rng.random(), 5)}
    if kind == "particles":
        n = rng.choice((48, 64, 96, 128, 256, 512))
        return {"kind": kind, "n": n, "prec": prec, "particles": int(10 ** (3 + 3 * rng.random())) | 1,
                "steps": rng.randint(4, 30)}
    n = rng.choice(SIZES[:-1])
    nc = rng.choice((0, 0, 1))
    rk = 4 if nc == 0 and rng.random() < 0.25 else 2
    np_ = int(10 ** (2 + 3 * rng.random())) | 1 if rk == 2 and rng.random() < 0.3 else 0
    return {"kind": "run", "n": n, "steps": rng.randint(3, 20) if n <= 256 else rng.randint(3, 6), "prec": prec,
            "nc": nc, "rk": rk, "particles": np_, "forced": False,
            # adaptive dt only where few passes are made: a small unforced box stepped for ever decays, and
            # its time step would grow without bound
            "dt": round((0.1 + 0.2 * rng.random()) / n, 6) if n < 256 or rng.random() < 0.3 else 0.0,
            "kshift": rng.choice((1, 2, 3, 4))}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def viscosity(n):
    """kmax eta near 1.5 for the unit-velocity field above."""
    return 0.6 * (2.0 / n) ** (4.0 / 3.0)


def columns(n):
    """The (kx, kz) columns of the truncation cylinder in the state's order, the entries inside the
    truncation sphere [columns, n], and the number of kx kept."""
    kxn = min(n // 2, math.isqrt(2 * n * n // 9) + 1)
    xs, zs = [], []
    for x in range(kxn):
        c = int(n * (1.0 - 2.0 * math.sqrt(2.0 / 9.0 - (x / n) ** 2)) / 2)
        kc = n // 2 - 1 - c
        kz = list(range(kc + 1)) + list(range(-kc, 0))
        xs += [x] * len(kz)
        zs += kz
    xs, zs = np.array(xs), np.array(zs)
    ky = np.fft.fftfreq(n, 1.0 / n)
    inside = ((ky / n) ** 2)[None, :] + ((zs / n) ** 2 + (xs / n) ** 2)[:, None] <= 2.0 / 9.0
    inside[:, n // 2] = False
    return xs, zs, inside


class Waves:
    """Wavenumbers and the sphere mask of the half-complex arrays [z, y, x] in FP64."""

    def __init__(self, n):
        self.n = n
        full = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
        full[n // 2] = n // 2
        self.kx = torch.arange(n // 2 + 1, dtype=torch.float64, device="cuda")[None, None, :]
        self.ky = full[None, :, None]
        self.kz = full[:, None, None]
        xs, zs, inside = columns(n)
        self.zi = torch.from_numpy(zs % n).cuda()
        self.xi = torch.from_numpy(xs).cuda()
        m = torch.zeros(n, n, n // 2 + 1, dtype=torch.bool, device="cuda")
        m[self.zi, :, self.xi] = torch.from_numpy(inside).cuda()
        self.mask = m

    def k2(self):
        return self.kx ** 2 + self.ky ** 2 + self.kz ** 2

    def project(self, u):
        k2 = self.k2()
        k2[0, 0, 0] = 1.0
        s = (self.kx * u[0] + self.ky * u[1] + self.kz * u[2]) / k2
        s[0, 0, 0] = 0.0
        return [u[0] - self.kx * s, u[1] - self.ky * s, u[2] - self.kz * s]

    def to_columns(self, fields):
        """[v][z, y, x] -> the state layout [v, column, y]."""
        return torch.stack([f[self.zi, :, self.xi] for f in fields])


def field(w, seed, nc=0):
    """The initial field in FP64: a list of 3 + nc half-complex arrays."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n = w.n
    k = w.k2().sqrt()
    k[0, 0, 0] = 1.0
    ek = k ** 4 * (1.0 + (k / 3.0) ** 2) ** (-17.0 / 6.0) * torch.exp(-4.0 * k / (n * math.sqrt(2.0) / 3.0))
    amp = torch.where(w.mask, (ek / k ** 2).sqrt(), torch.zeros_like(k))
    amp[0, 0, 0] = 0.0
    out = [torch.fft.rfftn(torch.randn(n, n, n, dtype=torch.float64, device="cuda", generator=g)) * amp
           for _ in range(3 + nc)]
    out[:3] = w.project(out[:3])
    two = torch.full((n // 2 + 1,), 2.0, dtype=torch.float64, device="cuda")
    two[0] = 1.0
    e = sum((two * (f.real ** 2 + f.imag ** 2)).sum() for f in out[:3])
    scale = (3.0 / e).sqrt()
    return [f * scale for f in out]


def particle_positions(n, count, seed):
    return 1.0 + n * np.random.default_rng(seed).random((count, 3))


def box_options(case):
    n = case["n"]
    kw = {"n": n, "precision": P.PREC_FP64 if case["prec"] == "fp64" else P.PREC_FP32,
          "viscos": case.get("nu", viscosity(n)), "kshift": case.get("kshift", 1), "nc": case.get("nc", 0),
          "cfl": -1.0, "dt": 0.25 / n}
    if case["kind"] == "run":
        # dt = 0: adaptive, at Courant number 0.5 (cfl = pi); RK4 runs use the larger number of the shipped input
        kw.update({"cfl": -1.0, "dt": case["dt"]} if case["dt"] else
                  {"cfl": 3.77 if case["rk"] == 4 else math.pi, "dt": 0.0})
        kw["rkmethod"] = case["rk"]
        if case["nc"]:
            kw.update(pr=1.0, grad=(1.0, 0.0, 0.0))
        if case["forced"]:
            kw.update(kforce=2.99, tforce=0.5, epsfor=0.1 / (4.0 * (4.0 * math.pi / 3.0) * 27.0), tfiuo=0.0)
    return kw


def ensemble_boxes(case, seed):
    """(n, viscosity, seed of the field) of every box: `pick` says which sizes, the seed which fields."""
    r = np.random.default_rng(case["pick"])
    ns = [int(v) for v in r.choice(ENSEMBLE_SIZES, case["boxes"])]
    nus = [float(v) for v in np.exp(r.uniform(math.log(0.005), math.log(0.05), case["boxes"]))]
    return [(n, nu, 1000 * (seed % 1000003) + i) for i, (n, nu) in enumerate(zip(ns, nus))]


class State:
    """A handle and the pinned host array that its state is written to."""

    def __init__(self, case):
        self.case, self.solver, self.host, self.ptr = case, None, None, None

    def pin(self, shape):
        self.host = np.zeros(shape, np.complex128)
        self.ptr = P.host_register(self.host)

    def __del__(self):
        if self.solver is not None:
            self.solver.close()
        if self.ptr is not None:
            P.host_unregister(self.host)


def prepare(case, seed):
    s = State(case)
    if case["kind"] == "ensemble":
        boxes = ensemble_boxes(case, seed)
        prec = P.PREC_FP64 if case["prec"] == "fp64" else P.PREC_FP32
        s.solver = P.Ensemble([P.default_params(n=n, precision=prec, viscos=nu, cfl=-1.0, dt=0.005, kshift=1,
                                                seed_input=1000 + i) for i, (n, nu, _) in enumerate(boxes)])
        waves = {n: Waves(n) for n in {b[0] for b in boxes}}
        for i, (n, _, fs) in enumerate(boxes):
            s.solver.set_state(i, waves[n].to_columns(field(waves[n], fs)).cpu().numpy())
        s.solver.step(ENSEMBLE_WARM)
        return s
    n = case["n"]
    if case["kind"] == "stage":
        w = Waves(n)
        s.params = P.default_params(**box_options(case))
        s.un = w.to_columns(field(w, seed))
        if case["prec"] == "fp32":
            s.un = s.un.to(torch.complex64)
        s.u = s.un.clone()
        s.gsh = np.random.default_rng(seed).random((3, 2))
        return s
    s.solver = P.Solver(**box_options(case))
    if n == 1024:
        # the library's own random field: one made in FP64 with torch does not fit beside three boxes
        s.solver.field_init(1 + seed % 2000000000)
    else:
        w = Waves(n)
        s.solver.set_state(w.to_columns(field(w, seed, case.get("nc", 0))).cpu().numpy())
        del w
        torch.cuda.empty_cache()
    if case.get("particles"):
        s.solver.particles_set(particle_positions(n, case["particles"], seed))
    if case["kind"] == "run":
        s.pin(s.solver.state_shape())
    s.gsh = np.random.default_rng(seed).random(3)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "stage":
        dt = s.params.dt
        stream = torch.cuda.current_stream().cuda_stream
        vm = P.rk_stage_noalloc(s.params, 1, s.gsh, dt, s.u.data_ptr(), s.un.data_ptr(), stream)
        P.rk_stage_noalloc(s.params, 2, s.gsh, dt, s.u.data_ptr(), s.un.data_ptr(), stream)
        return {"un": s.un, "velmax": float(vm)}
    b = s.solver
    if kind == "run":
        for _ in range(case["steps"]):
            info = b.step()
        b.get_state_sphere_async_ptr(s.ptr)
        b.sync()
        out = {"un": torch.from_numpy(s.host), "dt": float(info["dt"]), "velmax": float(info["velmax"])}
        if case["particles"]:
            out["pos"], out["vel"] = b.particles_get()
        return out
    if kind == "particles":
        for _ in range(case["steps"]):
            b.particles_advance(s.gsh, 0.25 / case["n"])
        pos, vel = b.particles_get()
        return {"pos": pos, "vel": vel}
    if kind == "diagnostics":
        ek, dk, eij, _ = b.spectra()
        xr, yr, zr, _ = b.spectra_scales()
        ux, wz = b.gradient_moments(gsh=s.gsh)
        return {"ek": ek, "dk": dk, "eij": eij, "xr": xr, "yr": yr, "zr": zr, "ux": ux, "wz": wz,
                "tk": b.transfer_spectrum(gsh=s.gsh)}
    b.step(case["steps"])
    return [b.get_state(i) for i in range(case["boxes"])]


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how far another correct program may be off
# ---------------------------------------------------------------------------
def work(case):
    size = 16 if case["prec"] == "fp64" else 8

    def modes(n):
        return 2.0 / 3.0 * math.pi * (math.sqrt(2.0) / 3.0 * n) ** 3   # half of the truncation sphere

    def fft(n):
        return 2.5 * n ** 3 * math.log2(n ** 3)                         # one real 3-D transform

    def stage(n, nc=0):
        # u and un in and out; 3 + 3 nc transforms back and 5 + nc forward
        return 4 * (3 + nc) * modes(n) * size, (8 + 4 * nc) * fft(n)

    def particle(n, count):
        return 3 * modes(n) * size + 96.0 * count, 3 * fft(n) + 2 * 64 * 6.0 * count

    kind = case["kind"]
    if kind == "ensemble":
        s = [stage(b[0]) for b in ensemble_boxes(case, 0)]
        by, fl = (2 * case["steps"] * sum(v[i] for v in s) for i in (0, 1))
        return {"bytes": by + sum(48 * modes(b[0]) for b in ensemble_boxes(case, 0)), "flops": fl}
    n = case["n"]
    if kind == "stage":
        by, fl = stage(n)
        return {"bytes": 2 * by, "flops": 2 * fl}
    if kind == "run":
        by, fl = stage(n, case["nc"])
        pb, pf = particle(n, case["particles"]) if case["particles"] else (0.0, 0.0)
        out = 16 * (3 + case["nc"]) * modes(n) + 48.0 * case["particles"]
        return {"bytes": case["steps"] * (case["rk"] * by + pb) + out, "flops": case["steps"] * (case["rk"] * fl + pf)}
    if kind == "particles":
        pb, pf = particle(n, case["particles"])
        return {"bytes": case["steps"] * pb + 48.0 * case["particles"], "flops": case["steps"] * pf}
    # the state once for each of the four, the transforms of the gradients and of the convective term
    return {"bytes": 4 * 3 * modes(n) * size, "flops": 10 * fft(n) + 100 * modes(n)}


def tolerance(case):
    """About four times what the results are off exact(): FP32 fields are 5e-8 off after a step and up to 8e-7
    after twenty (advection terms, moments and velocities 5e-7 to 1.1e-6), an ensemble's 1e-5 after its
    hundreds of steps; FP64 ones 2e-15."""
    long_ = case["kind"] == "ensemble"
    if case["prec"] == "fp64":
        return {"rel": 2e-13 if long_ else 1e-14, "max": 1e-10}
    return {"rel": 5e-5 if long_ else 4e-6, "max": 5e-3 if long_ else 1e-3}


# ---------------------------------------------------------------------------
# the same results in FP64 with torch
# ---------------------------------------------------------------------------
class Shifts:
    """Grid shifts of the run's random sequence: s <- 65539 s mod 2^31, six draws a step."""

    def __init__(self, kshift, seed=122929298):
        self.s, self.k, self.first, self.g = seed, kshift, True, [[0.0, 0.0] for _ in range(6)]

    def draw(self):
        self.s = self.s * 65539 % 2 ** 31
        return self.s * 0.46566127e-9

    def step(self):
        if self.first and self.k in (1, 3):
            for g in self.g:
                g[1] = self.draw()
        self.first = False
        other = lambda v: math.fmod(v + 0.5, 1.0)  # noqa: E731
        for g in self.g:
            if self.k == 1:
                g[0], g[1] = other(g[1]), self.draw()
            elif self.k == 2:
                g[0] = self.draw()
                g[1] = other(g[0])
            elif self.k == 3:
                g[0] = other(g[1])
                g[1] = other(g[0])
        return [[self.g[i][0] for i in range(3)], [self.g[i][1] for i in range(3)]]


class Exact:
    """One box in FP64: fields un, u and the accumulator of RK4 as half-complex arrays [z, y, x]."""

    def __init__(self, w, un, nu, nc=0, grad=(1.0, 0.0, 0.0)):
        self.w, self.nu, self.nc, self.grad = w, nu, nc, grad
        self.un, self.u = un, [f.clone() for f in un]
        self.vel = None

    def shift(self, g):
        w = self.w
        return torch.exp(1j * (2.0 * math.pi / w.n) * (w.kx * g[0] + w.ky * g[1] + w.kz * g[2]))

    def grid(self, f):
        n = self.w.n
        return torch.fft.irfftn(f, s=(n, n, n), norm="forward")

    def terms(self, fields, g):
        """(N(u) of every variable, velmax) with N the advection terms on the grid shifted by g."""
        w = self.w
        sh = torch.where(w.mask, self.shift(g), torch.zeros((), dtype=torch.complex128, device="cuda"))
        ug = [self.grid(f * sh) for f in fields[:3]]
        vmax = w.n * float((ug[0].abs() + ug[1].abs() + ug[2].abs()).max())
        back = sh.conj()
        k = (w.kx, w.ky, w.kz)
        out = [None, None, None]
        for i in range(3):
            for j in range(i, 3):
                t = torch.fft.rfftn(ug[i] * ug[j], norm="forward") * back
                for a, b in ((i, j), (j, i)) if i != j else ((i, j),):
                    d = (-1j) * k[b] * t
                    out[a] = d if out[a] is None else out[a] + d
        if self.nc:
            th = fields[3] * sh
            s = sum(ug[a] * (self.grad[a] + self.grid(1j * k[a] * th)) for a in range(3))
            out.append(-torch.fft.rfftn(s, norm="forward") * back)
        return out, vmax

    def clean(self, f):
        f = [torch.where(self.w.mask, v, torch.zeros_like(v)) for v in f]
        f[:3] = self.w.project(f[:3])
        return f

    def step(self, gsh, dt=None, cfl=0.0, rk=2):
        """One step with the shifts gsh of its stages; returns (dt, velmax)."""
        n, vmax = range(3 + self.nc), None
        for k in range(rk):
            t, v = self.terms(self.u, gsh[k % 2])
            if k == 0:
                vmax = v
                dt = cfl / v if cfl > 0 else dt
                f = torch.exp(-self.nu * dt * self.w.k2())
            t = [v * (0.5 * dt) for v in t]
            if rk == 2 and k == 0:
                self.u = self.clean([f * (self.un[i] + 2.0 * t[i]) for i in n])
                self.un = [torch.where(self.w.mask, f * (self.un[i] + t[i]), torch.zeros_like(t[i])) for i in n]
            elif rk == 2:
                self.u = self.clean([self.un[i] + t[i] for i in n])
                for v in self.u:
                    v[0, 0, 0] = 0.0
                self.un = [v.clone() for v in self.u]
            elif k == 0:
                acc = [f * (self.un[i] + t[i] / 3.0) for i in n]
                self.u = self.clean([f * (self.un[i] + t[i]) for i in n])
            elif k < 3:
                acc = [acc[i] + t[i] * (2.0 / 3.0) for i in n]
                self.u = self.clean([self.un[i] + t[i] * float(k) for i in n])
            else:
                self.u = self.clean([acc[i] + t[i] / 3.0 for i in n])
                for v in self.u:
                    v[0, 0, 0] = 0.0
                self.un = [v.clone() for v in self.u]
        return dt, vmax

    def spline(self, g):
        """Cubic B-spline coefficients of the velocity on the grid shifted by g."""
        w, n = self.w, self.w.n
        h = lambda k: 6.0 / (4.0 + 2.0 * torch.cos(2.0 * math.pi * k / n))  # noqa: E731
        f = torch.where(w.mask, self.shift(g), torch.zeros((), dtype=torch.complex128, device="cuda"))
        f = f * h(w.kx) * h(w.ky) * h(w.kz)
        return [self.grid(v * f).reshape(-1) for v in self.u[:3]]

    def interpolate(self, coef, pos, g):
        n = self.w.n
        at = pos - 1.0 - torch.tensor(g, dtype=torch.float64, device="cuda")
        i0 = torch.floor(at)
        t = at - i0
        i0 = i0.to(torch.int64)
        m = 1.0 - t
        ws = [m ** 3 / 6.0, 2.0 / 3.0 + 0.5 * t * (m * m - 1.0), None, t ** 3 / 6.0]
        ws[2] = 1.0 - ws[0] - ws[1] - ws[3]
        out = torch.zeros_like(pos)
        for kz in range(4):
            for ky in range(4):
                for kx in range(4):
                    j = [(i0[:, a] + k - 1) % n for a, k in enumerate((kx, ky, kz))]
                    idx = (j[2] * n + j[1]) * n + j[0]
                    wt = ws[kx][:, 0] * ws[ky][:, 1] * ws[kz][:, 2]
                    for c in range(3):
                        out[:, c] += wt * coef[c][idx]
        return out

    def particles(self, pos, g, dt):
        """Heun step of the positions with the previous step's dt; the first call only interpolates."""
        coef = self.spline(g)
        if self.vel is not None:
            f = 0.5 * dt / 2.0 / math.pi * self.w.n
            half = pos + f * self.vel
            pos = half + f * self.interpolate(coef, half + f * self.vel, g)
        self.vel = self.interpolate(coef, pos, g)
        return pos


def exact_diagnostics(case, seed):
    n, nu = case["n"], case.get("nu", viscosity(case["n"]))
    w = Waves(n)
    box = Exact(w, field(w, seed), nu)
    g = [float(v) for v in np.random.default_rng(seed).random(3)]
    two = torch.full((1, 1, n // 2 + 1), 2.0, dtype=torch.float64, device="cuda")
    two[..., 0] = 1.0
    un = w.to_columns(box.un)
    x, z = w.xi, torch.from_numpy(columns(n)[1]).cuda()
    ky = w.ky[0, :, 0]
    tf = torch.where(x == 0, 1.0, 2.0).double()[:, None]
    k2 = (x.double() ** 2 + z.double() ** 2)[:, None] + ky[None, :] ** 2
    ik = (k2.sqrt() + 1.5).to(torch.int64) - 1
    inside = torch.from_numpy(columns(n)[2]).cuda()

    def shells(v, length):
        v = torch.where(inside, v, torch.zeros_like(v))
        ok = ik < length
        return torch.zeros(length, dtype=torch.float64, device="cuda").index_add_(0, ik[ok], v[ok])

    pairs = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
    prod = [(un[i] * un[j].conj()).real for i, j in pairs]
    tr = prod[0] + prod[3] + prod[5]
    ek = 0.5 * shells(tf * tr, n)
    dk = nu * shells(tf * k2 * tr, n)
    ek[0] = dk[0] = 0.0
    eij = torch.stack([shells(tf * p, n) for p in prod], 1)
    nh = n // 2 + 1
    ones = []
    for p in prod:
        p = torch.where(inside, p, torch.zeros_like(p))
        zero = lambda: torch.zeros(nh, dtype=torch.float64, device="cuda")  # noqa: E731
        col = p.sum(1)
        fold = torch.where(tf[:, 0] > 1.0, 1.0, 0.0).double()
        xr = zero().index_add_(0, x, col)
        yr = zero()
        cols = (p * torch.where(ky[None, :] == 0, tf, torch.where(ky[None, :] > 0, torch.ones_like(tf),
                                                                    fold[:, None]))).sum(0)
        yr.index_add_(0, ky.abs().to(torch.int64), cols)
        wz = torch.where(z == 0, tf[:, 0], torch.where(z > 0, torch.ones_like(fold), fold))
        zr = zero().index_add_(0, z.abs(), col * wz)
        ones.append((xr, yr, zr))
    sh = box.shift(g)
    mom = []
    for f, k in ((box.un[0], w.kx), (box.un[2], w.kz)):
        v = box.grid(1j * k * f * sh)
        mom.append(torch.stack([(v ** m).mean() for m in range(1, 9)]))
    t, _ = box.terms(box.u, g)
    t = w.to_columns(t)
    tk = shells(tf * sum((un[i].conj() * t[i]).real for i in range(3)), n // 2)
    return {"ek": ek, "dk": dk, "eij": eij, "xr": torch.stack([o[0] for o in ones]),
            "yr": torch.stack([o[1] for o in ones]), "zr": torch.stack([o[2] for o in ones]),
            "ux": mom[0], "wz": mom[1], "tk": tk}


def exact(case, seed):
    kind = case["kind"]
    if kind == "diagnostics":
        return exact_diagnostics(case, seed)
    if kind == "ensemble":
        out, waves = [], {}
        for i, (n, nu, fs) in enumerate(ensemble_boxes(case, seed)):
            w = waves.setdefault(n, Waves(n))
            box, sh = Exact(w, field(w, fs), nu), Shifts(1, 1000 + i)
            for _ in range(ENSEMBLE_WARM + case["steps"]):
                box.step(sh.step(), dt=0.005)
            out.append(w.to_columns(box.un).cpu())
        return out
    n = case["n"]
    if n == 1024:
        return None   # over 20 seconds with the state's way to the host
    w = Waves(n)
    nc = case.get("nc", 0)
    box = Exact(w, field(w, seed, nc), case.get("nu", viscosity(n)), nc)
    if kind == "stage":
        gsh = np.random.default_rng(seed).random((3, 2))
        _, vm = box.step([list(gsh[:, 0]), list(gsh[:, 1])], dt=0.25 / n)
        return {"un": w.to_columns(box.un), "velmax": vm}
    pos = torch.from_numpy(particle_positions(n, case["particles"], seed)).cuda() if case["particles"] else None
    if kind == "particles":
        g = [float(v) for v in np.random.default_rng(seed).random(3)]
        for _ in range(case["steps"]):
            pos = box.particles(pos, g, 0.25 / n)
        return {"pos": pos, "vel": box.vel}
    sh, dt = Shifts(case["kshift"]), 0.0
    cfl = 0.0 if case["dt"] else (3.77 if case["rk"] == 4 else math.pi)
    for _ in range(case["steps"]):
        g = sh.step()
        if pos is not None:
            pos = box.particles(pos, g[0], dt)
        dt, vm = box.step(g, dt=case["dt"], cfl=cfl, rk=case["rk"])
    out = {"un": w.to_columns(box.un), "dt": dt, "velmax": vm}
    if pos is not None:
        out["pos"], out["vel"] = pos, box.vel
    return out
