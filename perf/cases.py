"""Performance cases of the solver: what a user's program has it do.

`listed()` names the cases, `draw(rng)` gives further ones of the same
ranges, `prepare(case, seed)` builds what the program has in hand (a set-up
context, host fields), `run(state)` makes one pass through the public entry
points and returns what it computed, `work(case)` says what the pass cannot
do without, and `exact(case, seed)` evaluates the same outputs in FP64 with
dense transform matrices (torch only; None where there is no such value).

Outputs of the FP64 form come as the entry points return them.  The mixed
form's transforms and products are FP32, so its fields are handed on as a
single-precision field file holds them; the host-owned state of
`advance_host` stays the FP64 array that the program owns.
"""
import math

import numpy as np
import torch

from ps3d_gb300 import Ps3dGpu, batch_advance
from ps3d_gb300.closure import Closure, attach
from ps3d_gb300.solver import PinnedArray

LOWER = (0.0, 0.0, -0.5 * math.pi)
EXTENT = (2.0 * math.pi, 2.0 * math.pi, math.pi)

# grid lengths the library takes: even, prime factors 2, 3 and 5
LENGTHS = sorted(2 ** a * 3 ** b * 5 ** c for a in range(1, 12) for b in range(5) for c in range(4)
                 if 8 <= 2 ** a * 3 ** b * 5 ** c <= 1024)


# ------------------------------------------------------------------ cases
def listed():
    return [
        # the small FP64 verification run (32^3, 200 steps in all): field
        # output every 20 steps; launches and latency count
        {"name": "fp64 32^3 run", "kind": "run", "form": "fp64", "nx": 32, "ny": 32, "nz": 32, "steps": 20,
         "stepper": "impl-diff-rk4", "pretype": "vorch", "filtering": "Hou & Li"},
        # the FP64 production size of the reference's own runs
        {"name": "fp64 128^3 run", "kind": "run", "form": "fp64", "nx": 128, "ny": 128, "nz": 128, "steps": 5,
         "stepper": "impl-diff-rk4", "pretype": "vorch", "filtering": "Hou & Li"},
        # a ragged box with factors 3 and 5, the other stepper, filter and
        # prefactor
        {"name": "fp64 96x160x60 cn2 run", "kind": "run", "form": "fp64", "nx": 96, "ny": 160, "nz": 60, "steps": 5,
         "stepper": "cn2", "pretype": "roll-mean-max-strain", "filtering": "2/3-rule"},
        # a stratified run (buoyancy stepped with the vorticity)
        {"name": "fp64 64x48x80 buoyancy run", "kind": "buoyancy", "form": "fp64", "nx": 64, "ny": 48, "nz": 80,
         "steps": 5, "stepper": "impl-diff-rk4"},
        # a Fortran driver that owns the FP64 state on the host: one advance
        # per call, state in and out of page-locked memory
        {"name": "fp64 256^3 host step", "kind": "host", "form": "fp64", "nx": 256, "ny": 256, "nz": 256},
        # the same driver at the headline size with the mixed form
        {"name": "mixed 512^3 host step", "kind": "host", "form": "mixed", "nx": 512, "ny": 512, "nz": 512},
        # captured mixed steps at the usual resolution, output every 50 steps
        {"name": "mixed 128^3 captured", "kind": "captured", "form": "mixed", "nx": 128, "ny": 128, "nz": 128,
         "steps": 50},
        # an ensemble of independent runs of uneven sizes in one batch
        {"name": "mixed batch of 12", "kind": "batch", "n32": 6, "n64": 4, "n128": 2, "steps": 20},
        # a coarse run with the learned closure evaluated at every stage
        {"name": "closure 64^3 captured", "kind": "closure", "nx": 64, "ny": 64, "nz": 64, "steps": 20},
        # training that closure: Adam steps over stored samples
        {"name": "closure 64^3 training", "kind": "training", "nx": 64, "ny": 64, "nz": 64, "samples": 4,
         "iters": 20},
        # a single field operator called on a host array (initialisation,
        # analysis); the smallest call
        {"name": "fp64 32^3 decompose", "kind": "operator", "form": "fp64", "op": "decompose_physical", "nx": 32,
         "ny": 32, "nz": 32},
        # standalone inversion of a K^(-5/3) spectral vorticity, and the
        # quantities written at an output time
        {"name": "fp64 128^3 inversion", "kind": "inversion", "form": "fp64", "nx": 128, "ny": 128, "nz": 128},
    ]


def _length(rng, lo, hi):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min((n for n in LENGTHS if lo <= n <= hi), key=lambda n: abs(math.log(n / v)))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "host", "host", "captured", "batch", "buoyancy", "closure", "training",
                       "operator", "inversion"])
    form = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        return {"kind": kind, "n32": rng.randint(1, 12), "n64": rng.randint(0, 6), "n128": rng.randint(0, 3),
                "steps": rng.randint(5, 20)}
    lo, hi = {"run": (16, 192), "host": (48, 288), "captured": (24, 192), "buoyancy": (24, 128), "closure": (12, 96),
              "training": (12, 80), "operator": (16, 192), "inversion": (24, 192)}[kind]
    c = {"kind": kind, "nx": _length(rng, lo, hi), "ny": _length(rng, lo, hi), "nz": _length(rng, lo, hi)}
    if kind in ("closure", "training"):  # the closure's grids are powers of two
        c.update({k: 2 ** round(math.log2(c[k])) for k in ("nx", "ny", "nz")})
    small = c["nx"] * c["ny"] * c["nz"] < 100 ** 3
    if kind in ("run", "buoyancy"):
        c.update(form=form, steps=rng.randint(2, 12 if small else 4),
                 stepper=rng.choice(["impl-diff-rk4", "impl-diff-rk4", "cn2"]))
    if kind == "run":
        c.update(pretype=rng.choice(["constant", "vorch", "max-strain", "roll-mean-max-strain"]),
                 filtering=rng.choice(["Hou & Li", "2/3-rule"]))
    if kind in ("host", "operator", "inversion"):
        c.update(form=form)
    if kind == "operator":
        c.update(op=rng.choice(["decompose_physical", "combine_physical", "fftxyp2s", "fftsine", "diffx"]))
    if kind in ("captured", "closure"):
        c.update(form="mixed", steps=rng.randint(4, 30))
    if kind == "training":
        c.update(samples=rng.randint(1, 4), iters=rng.randint(4, 20))
    return c


# ---------------------------------------------------------------- inputs
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _wavenumbers(n, length, periodic):
    if not periodic:
        return math.pi / length * torch.arange(n + 1, dtype=torch.float64, device="cuda")
    k = torch.arange(n, dtype=torch.float64, device="cuda")
    return 2.0 * math.pi / length * torch.minimum(k, n - k)


def _k2(nx, ny, nz):
    kx, ky = _wavenumbers(nx, EXTENT[0], True), _wavenumbers(ny, EXTENT[1], True)
    kz = _wavenumbers(nz, EXTENT[2], False)
    return kx[:, None, None] ** 2 + ky[None, :, None] ** 2 + kz[None, None, :] ** 2


def _beltrami(nx, ny, nz):
    """(3, nx, ny, nz+1) vorticity of the Beltrami flow k = l = 2, m = 1"""
    ar = lambda n: torch.arange(n, dtype=torch.float64, device="cuda")  # noqa: E731
    x = EXTENT[0] / nx * ar(nx)
    y = EXTENT[1] / ny * ar(ny)
    z = LOWER[2] + EXTENT[2] / nz * ar(nz + 1)
    ph = 2.0 * x[:, None, None] + 2.0 * y[None, :, None]
    g = torch.stack([(2.0 * torch.sin(z) - 6.0 * torch.cos(z)) * 3.0 / 8.0,
                     (2.0 * torch.sin(z) + 6.0 * torch.cos(z)) * 3.0 / 8.0, 3.0 * torch.cos(z)])
    return torch.stack([torch.sin(ph) * g[0], torch.sin(ph) * g[1], torch.cos(ph) * g[2]])


def _perturbation(nx, ny, nz, gen, amplitude, rms):
    """Gaussian spectral vorticity with a K^-2 envelope in the interior sine
    modes, grid rms amplitude * rms by Parseval"""
    env = 1.0 / _k2(nx, ny, nz).clamp_min(1e-3)
    env[:, :, 0] = 0.0
    env[:, :, nz] = 0.0
    env[nx // 2] = 0.0
    env[:, ny // 2] = 0.0
    p = torch.randn((3, nx, ny, nz + 1), dtype=torch.float64, device="cuda", generator=gen) * env
    wx = torch.full((nx, 1, 1), 2.0, dtype=torch.float64, device="cuda")
    wy = torch.full((ny, 1), 2.0, dtype=torch.float64, device="cuda")
    wx[0] = wx[nx // 2] = wy[0] = wy[ny // 2] = 1.0
    ms = float((p.square().sum(0) * wx * wy).sum()) / (nx * ny * (nz + 1))
    return p * (amplitude * rms / math.sqrt(ms))


def _flow(c, seed, amplitude=1.0e-2):
    gen = _generator(seed)
    vor = _beltrami(c["nx"], c["ny"], c["nz"])
    rms = float(vor.square().sum(0).mean().sqrt())
    return vor, _perturbation(c["nx"], c["ny"], c["nz"], gen, amplitude, rms)


def _kolmogorov(c, seed):
    """seeded spectral vorticity with a K^(-5/3) amplitude spectrum"""
    k2 = _k2(c["nx"], c["ny"], c["nz"])
    amp = torch.where(k2 > 0, k2.clamp_min(1e-3) ** (-5.0 / 6.0), torch.zeros_like(k2))
    gen = _generator(seed)
    p = torch.rand((3,) + tuple(k2.shape), dtype=torch.float64, device="cuda", generator=gen)
    f = amp * torch.cos(2.0 * math.pi * p)
    return f / f.square().mean().sqrt()


def _smooth(c, seed, n=1):
    """n physical fields: a few low modes plus a little noise"""
    gen = _generator(seed)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    x = 2.0 * math.pi / nx * torch.arange(nx, dtype=torch.float64, device="cuda")[:, None, None]
    y = 2.0 * math.pi / ny * torch.arange(ny, dtype=torch.float64, device="cuda")[None, :, None]
    z = math.pi / nz * torch.arange(nz + 1, dtype=torch.float64, device="cuda")[None, None, :]
    out = []
    for _ in range(n):
        a = torch.randn(24, dtype=torch.float64, device="cuda", generator=gen).tolist()
        f = 1e-3 * torch.randn((nx, ny, nz + 1), dtype=torch.float64, device="cuda", generator=gen)
        for j in range(6):
            f += a[j] * torch.cos((1 + j % 3) * x + (j - 2) * y + a[6 + j]) * torch.cos((1 + j % 4) * z + a[12 + j])
        out.append(f)
    return torch.stack(out)


def _host(t):
    return t.cpu().numpy()


def _context(c, **kw):
    return Ps3dGpu(c["nx"], c["ny"], c["nz"], LOWER, EXTENT, precision=c["form"], cflmax=0.5, nnu=3,
                   prediss=kw.pop("prediss", 30.0), **kw)


class State:
    """what the program keeps between passes"""

    def __init__(self, case, **kw):
        self.case, self.t = case, 0.0
        self.__dict__.update(kw)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        runs = []
        amp = np.random.RandomState(seed % (1 << 31))
        for n, count in ((32, c["n32"]), (64, c["n64"]), (128, c["n128"])):
            for _ in range(count):
                d = {"nx": n, "ny": n, "nz": n, "form": "mixed"}
                g = _context(d, pretype="vorch", prediss=float(amp.choice([10.0, 30.0, 60.0, 90.0])))
                vor, pert = _flow(d, seed + 7 * len(runs), 10.0 ** amp.uniform(-4.0, -2.0))
                g.setup_fields(_host(vor), _host(pert))
                runs.append(g)
        return State(c, runs=runs, ts=[0.0] * len(runs))
    if kind == "training":
        cl = Closure(c["nx"], c["ny"], c["nz"], max_samples=c["samples"], seed=seed % 1000)
        for k in range(c["samples"]):
            f = _smooth(c, seed + k, 6)
            vor, vel = f[:3], f[3:]
            target = 0.1 * (torch.roll(vor, 1, 1) - vor) * vel.roll(1, 0)
            cl.add_sample(_host(vor), _host(vel), _host(target))
        return State(c, closure=cl)
    if kind == "operator":
        return State(c, g=_context(c), field=_host(_smooth(c, seed)[0]))
    if kind == "inversion":
        g = _context(c)
        g.set("svor", _host(_kolmogorov(c, seed)))
        return State(c, g=g)
    if kind == "buoyancy":
        g = _context(c, buoyancy=True, bfsq=1.0, buoy_pretype="bfmax", pretype="vorch", stepper=c["stepper"])
        vor, pert = _flow(c, seed)
        z = LOWER[2] + EXTENT[2] / c["nz"] * torch.arange(c["nz"] + 1, dtype=torch.float64, device="cuda")
        s = torch.sin(math.pi / c["nz"] * torch.arange(c["nz"] + 1, dtype=torch.float64, device="cuda"))
        g.setup_fields(_host(vor), _host(pert), _host(z + 1e-2 * s * _smooth(c, seed + 1)[0]))
        return State(c, g=g)
    kw = {k: c[k] for k in ("stepper", "pretype", "filtering") if k in c}
    g = _context(dict(c, form="mixed" if kind == "closure" else c["form"]), **kw)
    vor, pert = _flow(c, seed)
    g.setup_fields(_host(vor), _host(pert))
    if kind == "closure":
        cl = Closure(c["nx"], c["ny"], c["nz"], seed=seed % 1000)
        cl.scale = 0.01
        attach(g, cl, every_stage=True)
        return State(c, g=g, closure=cl)
    if kind == "host":
        pinned = PinnedArray((3,) + g.shape)
        pinned.array[...] = g.get("svor")
        return State(c, g=g, pinned=pinned)
    return State(c, g=g)


# ------------------------------------------------------------------- runs
class Owned(np.ndarray):
    """a view of page-locked memory that keeps its owner alive"""

    owner = None


def _owned(pinned):
    a = pinned.array.view(Owned)
    a.owner = pinned
    return a


def _field(case, a):
    """a field as the program hands it on (see the module docstring)"""
    return torch.from_numpy(a) if case.get("form") == "fp64" else torch.from_numpy(a).to(torch.float32)


def run(state):
    s, c = state, state.case
    kind = c["kind"]
    if kind == "run":
        s.t, diags = s.g.advance_n(s.t, c["steps"])
        return {"svor": _field(c, s.g.get("svor")), "t": s.t, "ke": diags[-1]["ke"], "en": diags[-1]["en"]}
    if kind == "buoyancy":
        s.t, diags = s.g.advance_n(s.t, c["steps"])
        return {"svor": _field(c, s.g.get("svor")), "sbuoy": _field(c, s.g.get("sbuoy")), "t": s.t}
    if kind == "host":
        s.t, diag = s.g.advance_host(s.pinned.array, s.t)
        return {"svor": _owned(s.pinned), "t": s.t, "ke": diag["ke"], "en": diag["en"]}
    if kind == "captured":
        s.t, diag, _ = s.g.advance_graph(s.t, c["steps"])
        return {"svor": _field(c, s.g.get("svor")), "t": s.t, "ke": diag["ke"], "en": diag["en"]}
    if kind == "closure":
        s.t, diag, _ = s.g.advance_graph(s.t, c["steps"])
        return {"svor": _field(c, s.g.get("svor")), "t": s.t}
    if kind == "batch":
        s.ts, _ = batch_advance(s.runs, s.ts, c["steps"])
        return {"svor": [_field(c, g.get("svor")) for g in s.runs], "t": list(s.ts)}
    if kind == "training":
        loss = s.closure.train(c["iters"])
        return {"params": s.closure.get_params(), "loss": loss.astype(np.float32)}
    if kind == "operator":
        return {c["op"]: _field(c, getattr(s.g, c["op"])(s.field))}
    s.g.vor2vel()
    return {"vel": _field(c, s.g.get("vel"))}


def work(case):
    """Per step and grid value: the fields that the stages of a step read and
    write, each once (FP64 1120 bytes, mixed 728; impl-diff-rk4), and the
    multiply-adds of its 49 three-dimensional transforms plus the pointwise
    terms; cn2 evaluates three right-hand sides instead of four."""
    c, kind = case, case["kind"]

    def step(nx, ny, nz, form, rhs=4):
        n = nx * ny * (nz + 1)
        return {"bytes": (1120.0 if form == "fp64" else 728.0) * n * rhs / 4,
                "flops": (49 * 2.5 * n * math.log2(nx * ny * nz) + 300.0 * n) * rhs / 4}

    def times(w, k):
        return {"bytes": w["bytes"] * k, "flops": w["flops"] * k}

    if kind == "batch":
        ws = [times(step(n, n, n, "mixed"), c["n%d" % n] * c["steps"]) for n in (32, 64, 128)]
        return {k: sum(w[k] for w in ws) for k in ("bytes", "flops")}
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    n = nx * ny * (nz + 1)
    size = 8 if c.get("form") == "fp64" else 4
    net = 2.0 * n * 27 * (6 * 32 + 32 * 32 + 32 * 32 + 32 * 3)
    if kind == "operator":
        return {"bytes": 16.0 * n, "flops": 2.5 * n * math.log2(nx * ny * nz)}
    if kind == "inversion":
        # svor read and written (projection), vor, vel and svel written; 10 transforms
        return {"bytes": 15.0 * size * n, "flops": 10 * 2.5 * n * math.log2(nx * ny * nz)}
    if kind == "training":
        # per step: sample read, activations of three hidden layers written and
        # read, forward and two backward products per layer
        return {"bytes": c["iters"] * n * (9 * 4 + 2 * 3 * 32 * 2.0), "flops": 3 * net * c["iters"]}
    w = step(nx, ny, nz, c.get("form", "mixed"), 3 if c.get("stepper") == "cn2" else 4)
    if kind == "buoyancy":
        w = times(w, 4.0 / 3.0)
    if kind == "closure":
        w = {"bytes": w["bytes"] + 4 * n * 2.0 * (16 + 3 * 2 * 32), "flops": w["flops"] + 4 * net}
    return times(w, c.get("steps", 1))


# ------------------------------------------------------------ FP64 values
class Plain:
    """The reference's right-hand side and steppers with dense transform
    matrices in FP64 (fields (nx, ny, nz+1), torch on the GPU)."""

    def __init__(self, c, prediss=30.0, cfl=0.5, nnu=3):
        self.c, self.nx, self.ny, self.nz = c, c["nx"], c["ny"], c["nz"]
        self.prediss, self.cfl, self.nnu = prediss, cfl, nnu
        nx, ny, nz = self.nx, self.ny, self.nz
        dev = dict(dtype=torch.float64, device="cuda")
        self.fx, self.ix = self._real_dft(nx)
        self.fy, self.iy = self._real_dft(ny)
        j = torch.arange(nz + 1, **dev)
        ang = torch.remainder(j[:, None] * j[None, :], 2 * nz) * (math.pi / nz)
        self.dst = torch.sin(ang) * math.sqrt(2.0 / nz)
        self.dst[0] = self.dst[nz] = 0.0
        self.dst[:, 0] = self.dst[:, nz] = 0.0
        self.dct = torch.cos(ang) * math.sqrt(2.0 / nz)
        self.dct[:, 0] *= 0.5
        self.dct[:, nz] *= 0.5
        self.dx = [EXTENT[0] / nx, EXTENT[1] / ny, EXTENT[2] / nz]
        kx, ky = _wavenumbers(nx, EXTENT[0], True), _wavenumbers(ny, EXTENT[1], True)
        kz = _wavenumbers(nz, EXTENT[2], False)
        self.rk = (kx, ky, kz)
        self.sx = (nx - torch.arange(nx, device="cuda")) % nx
        self.sy = (ny - torch.arange(ny, device="cuda")) % ny

        def coef(k, n):
            s = torch.where(torch.arange(n, device="cuda") > n // 2, 1.0, -1.0).to(k)
            s[0] = s[n // 2] = 0.0
            return s * k

        self.cx, self.cy = coef(kx, nx)[:, None, None], coef(ky, ny)[None, :, None]
        k2 = (kx[:, None] ** 2 + ky[None, :] ** 2)[:, :, None]
        self.k2 = k2
        self.ki = torch.where(k2 > 0, 1.0 / k2.clamp_min(1e-300), torch.zeros_like(k2))
        z = LOWER[2] + self.dx[2] * j
        zm, zp = (LOWER[2] + EXTENT[2] - z)[None, None], (z - LOWER[2])[None, None]
        kl = k2.sqrt()
        lz = EXTENT[2]
        ef = torch.exp(-kl * lz)
        div = 1.0 / (1.0 - ef * ef)
        half = 0.5 * self.ki
        q, r = div * (1.0 + ef * ef), div * 2.0 * ef
        lm, lp = kl * zm, kl * zp
        ep, em = torch.exp(-lp), torch.exp(-lm)
        phm, php = div * (ep - ef * em), div * (em - ef * ep)
        dphm, dphp = -kl * div * (ep + ef * em), kl * div * (em + ef * ep)
        self.thm, self.thp = half * (r * lm * php - q * lp * phm), half * (r * lp * phm - q * lm * php)
        self.dthm = -half * ((q * lp - 1.0) * dphm - r * lm * dphp)
        self.dthp = -half * ((q * lm - 1.0) * dphp - r * lp * dphm)
        phm[0, 0], php[0, 0] = zm[0, 0] / lz, zp[0, 0] / lz
        for f in (self.thm, self.thp, self.dthm, self.dthp):
            f[0, 0] = 0.0
        self.phm, self.php = phm, php
        self.green = -1.0 / (k2 + kz[None, None] ** 2).clamp_min(1e-300)
        self.green[:, :, 0] = -self.ki[:, :, 0]
        self.kz = kz
        self.gtop = 0.5 * lz * ((zp[0, 0] / lz) ** 2 - 1.0 / 3.0)
        self.gbot = self.gtop.flip(0)
        # horizontal filter, and the vertical factor of cn2
        if c.get("filtering", "Hou & Li") == "2/3-rule":
            cut = lambda k: (k <= 2.0 / 3.0 * k.max()).double()  # noqa: E731
            self.filt = (cut(kx)[:, None] * cut(ky)[None, :])[:, :, None]
            self.fz = cut(kz)
        else:
            cut = lambda k: -36.0 * (k / k.max()) ** 36  # noqa: E731
            self.filt = torch.exp(cut(kx)[:, None] + cut(ky)[None, :])[:, :, None]
            self.fz = torch.exp(cut(kz))
        self.filt[0, 0] = 1.0
        self.fz[0] = self.fz[nz] = 1.0
        self.hist = []

    @staticmethod
    def _real_dft(n):
        j = torch.arange(n, dtype=torch.float64, device="cuda")
        k = torch.minimum(j, n - j)
        a = torch.remainder(k[:, None] * j[None, :], n) * (2.0 * math.pi / n)
        f = torch.where((j <= n // 2)[:, None], torch.cos(a), -torch.sin(a)) / math.sqrt(n)
        w = torch.full((n,), 2.0, dtype=torch.float64, device="cuda")
        w[0] = w[n // 2] = 1.0
        return f, (f * w[:, None]).t().contiguous()

    def _xy(self, mx, my, f):
        g = torch.matmul(my, f)
        return torch.matmul(mx, g.reshape(self.nx, -1)).reshape(f.shape)

    def fwd(self, f):
        return self._xy(self.fx, self.fy, f)

    def inv(self, f):
        return self._xy(self.ix, self.iy, f)

    def ddx(self, f):
        return self.cx * f[self.sx]

    def ddy(self, f):
        return self.cy * f[:, self.sy]

    def ddz(self, f):
        g = torch.empty_like(f)
        h = 1.0 / self.dx[2]
        g[..., 1:-1] = (f[..., 2:] - f[..., :-2]) * (0.5 * h)
        g[..., 0] = (f[..., 1] - f[..., 0]) * h
        g[..., -1] = (f[..., -1] - f[..., -2]) * h
        return g

    def dec(self, f):
        g = torch.matmul(f - (f[..., :1] * self.phm + f[..., -1:] * self.php), self.dst.t())
        g[..., 0], g[..., -1] = f[..., 0], f[..., -1]
        return g

    def com(self, f):
        g = torch.matmul(f, self.dst.t()) + f[..., :1] * self.phm + f[..., -1:] * self.php
        g[..., 0], g[..., -1] = f[..., 0], f[..., -1]
        return g

    def project(self, s):
        ds = self.ddx(s[1]) - self.ddy(s[0])
        es = self.dec(self.ddz(self.com(s[2])))
        a, b = self.ki * (self.ddx(es) + self.ddy(ds)), self.ki * (self.ddy(es) - self.ddx(ds))
        a[0, 0], b[0, 0] = s[0][0, 0], s[1][0, 0]
        return [a, b, s[2]]

    def vor2vel(self, s):
        self.s = s = self.project(s)
        cs = self.com(s[2])
        self.vor = [self.inv(self.com(s[0])), self.inv(self.com(s[1])), self.inv(cs)]
        ds = self.ddy(s[0]) - self.ddx(s[1])
        d0, dn = ds[..., :1], ds[..., -1:]
        g = self.green * ds
        g[..., 0] = g[..., -1] = 0.0
        w = torch.matmul(g, self.dst.t()) + d0 * self.thm + dn * self.thp
        w[..., 0] = w[..., -1] = 0.0
        es = d0 * self.dthm + dn * self.dthp + torch.matmul(self.kz * g, self.dct.t())
        a, b = s[0][0, 0], s[1][0, 0]
        rkzi = torch.where(self.kz > 0, 1.0 / self.kz.clamp_min(1e-300), torch.zeros_like(self.kz))
        rkzi[-1] = 0.0
        u, v = self.ki * (self.ddx(es) + self.ddy(cs)), self.ki * (self.ddy(es) - self.ddx(cs))
        u[0, 0] = self.dct @ (-rkzi * b) + b[-1] * self.gtop - b[0] * self.gbot
        v[0, 0] = self.dct @ (rkzi * a) - a[-1] * self.gtop + a[0] * self.gbot
        self.svel = [u, v, w]
        self.vel = [self.inv(f) for f in self.svel]
        return s

    def source(self):
        (u, v, w), (xi, eta, zeta) = self.vel, self.vor
        r, q, p = u * eta - v * xi, w * xi - u * zeta, v * zeta - w * eta
        gq, gp = self.dec(self.fwd(self.ddz(q))), self.dec(self.fwd(self.ddz(p)))
        r, q, p = (self.dec(self.fwd(f)) for f in (r, q, p))
        return [self.ddy(r) - gq, gp - self.ddx(r), self.ddx(q) - self.ddy(p)]

    def _mean(self, f):
        """grid sum over the cells (trapezoid in z) over their number"""
        return float((f[..., :-1] + f[..., 1:]).sum()) * 0.5 / (self.nx * self.ny * self.nz)

    def energies(self):
        return (0.5 * self._mean(sum(f * f for f in self.vel)), 0.5 * self._mean(sum(f * f for f in self.vor)))

    def setup(self, vor, pert):
        s = [self.dec(self.fwd(f)) for f in vor]
        self.state = [a + b for a, b in zip(s, pert)]
        self.ini = [self._col_mean(self.state[k]) for k in (0, 1)]
        self.state = self.vor2vel(self.state)
        ke, en = self.energies()
        k2max = max(float(k.max()) for k in self.rk[:2]) ** 2
        vis = self.prediss * (k2max * ke / en) ** (1.0 / 3.0) / k2max ** self.nnu
        self.hdis = vis * self.k2 ** self.nnu

    def _col_mean(self, f):
        c = f[0, 0]
        return 0.5 * (c[0] + c[-1]) + (self.dst @ c).sum() / self.nz

    def adapt(self, t):
        u, v, w = self.svel
        dudx, dudy, dwdx, dvdy, dwdy = (self.inv(f) for f in (self.ddx(u), self.ddy(u), self.ddx(w), self.ddy(v),
                                                              self.ddy(w)))
        xi, eta, zeta = self.vor
        a01, a02, a12 = dudy + 0.5 * zeta, dwdx + 0.5 * eta, dwdy - 0.5 * xi
        a22 = -(dudx + dvdy)
        s = (((dudx * dudx + dvdy * dvdy + a22 * a22) + 2.0 * (a01 * a01 + a02 * a02 + a12 * a12)) / 6.0).sqrt()
        det = (dudx * (dvdy * a22 - a12 * a12) - a01 * (a01 * a22 - a12 * a02) + a02 * (a01 * a12 - dvdy * a02))
        th = torch.acos((det / (2.0 * s ** 3).clamp_min(1e-300)).clamp(-1.0, 1.0)) / 3.0
        lam = torch.maximum((2.0 * s * torch.cos(th)).abs(), (2.0 * s * torch.cos(th + 2.0 * math.pi / 3.0)).abs())
        gg = float(lam.max())
        self.hist.append(gg)
        rms = math.sqrt(self._mean(xi * xi + eta * eta + zeta * zeta))
        mids = [0.5 * (f[..., :-1] + f[..., 1:]).abs() for f in self.vor]
        l1 = mids[0] + mids[1] + mids[2]
        l2 = mids[0] ** 2 + mids[1] ** 2 + mids[2] ** 2
        on = l1 > rms
        vorch = float(l2[on].sum()) / (1e-12 + float(l1[on].sum()))
        speed = [float(f.max()) for f in self.vel]
        dt = min(0.1 / (gg + 1e-12), self.cfl * min(h / (m + 1e-12) for h, m in zip(self.dx, speed)))
        pre = {"constant": 1.0, "vorch": vorch, "max-strain": gg,
               "roll-mean-max-strain": sum(self.hist) / len(self.hist)}[self.c.get("pretype", "vorch")]
        return dt, pre

    def _fix(self, s):
        for k in (0, 1):
            m = self.ini[k] - self._col_mean(s[k])
            s[k] = s[k].clone()
            s[k][0, 0, 0] += m
            s[k][0, 0, -1] += m
        return s

    def advance(self, t):
        q = self.vor2vel(self.state)
        self.series = self.energies()
        dt, pre = self.adapt(t)
        s = self.source()
        if self.c.get("stepper", "impl-diff-rk4") == "cn2":
            dis = 1.0 / (1.0 + pre * dt * self.hdis)
            f = self.filt * self.fz
            f[0, 0] = 1.0
            mid = [a + 0.5 * dt * b for a, b in zip(q, s)]
            for it in range(3):
                if it:
                    self.vor2vel(q)
                    s = self.source()
                q = self._fix([f * (a + 0.5 * dt * b) * dis for a, b in zip(mid, s)])
            self.state = q
            return t + dt
        e = torch.exp(0.5 * pre * dt * self.hdis)
        m, p = 1.0 / e, e * self.filt
        q0 = q
        s = [self.filt * a for a in s]
        acc = [a + dt / 6.0 * b for a, b in zip(q0, s)]
        q = [(a + 0.5 * dt * b) * m for a, b in zip(q0, s)]
        for step, fac in ((0.5 * dt, m), (dt, m * m)):
            self.vor2vel(q)
            s = [p * a for a in self.source()]
            q = [(a + step * b) * fac for a, b in zip(q0, s)]
            acc = [a + dt / 3.0 * b for a, b in zip(acc, s)]
        self.vor2vel(q)
        s = [p * p * a for a in self.source()]
        self.state = self._fix([(a + dt / 6.0 * b) * (m * m) for a, b in zip(acc, s)])
        return t + dt


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("buoyancy", "closure", "training"):
        return None  # no plain FP64 counterpart here
    if kind == "batch":
        return None if c["steps"] * c["n128"] > 60 else _exact_batch(c, seed)
    n = c["nx"] * c["ny"] * c["nz"]
    if n * c.get("steps", 1) > 1.4e8 or n > 3e7:
        return None  # over about 20 seconds
    if kind == "operator":
        p, f = Plain(c), _smooth(c, seed)[0]
        ops = {"decompose_physical": lambda: p.dec(p.fwd(f)), "combine_physical": lambda: p.inv(p.com(f)),
               "fftxyp2s": lambda: p.fwd(f), "diffx": lambda: p.ddx(f), "fftsine": lambda: _sine(p, f)}
        return {c["op"]: ops[c["op"]]()}
    if kind == "inversion":
        p = Plain(c)
        s = _kolmogorov(c, seed)
        p.vor2vel([s[0], s[1], s[2]])
        return {"vel": torch.stack(p.vel)}
    p = Plain(c)
    vor, pert = _flow(c, seed)
    p.setup(vor, pert)
    t = 0.0
    for _ in range(c.get("steps", 1)):
        t = p.advance(t)
    state = p.project(p.state) if c["form"] == "mixed" else p.state
    return {"svor": torch.stack(state), "t": t, "ke": p.series[0], "en": p.series[1]}


def _sine(p, f):
    g = torch.matmul(f, p.dst.t())
    g[..., 0] = f[..., 0]
    return g


def _exact_batch(c, seed):
    amp = np.random.RandomState(seed % (1 << 31))
    out, ts, k = [], [], 0
    for n, count in ((32, c["n32"]), (64, c["n64"]), (128, c["n128"])):
        for _ in range(count):
            d = {"nx": n, "ny": n, "nz": n, "form": "mixed"}
            p = Plain(d, prediss=float(amp.choice([10.0, 30.0, 60.0, 90.0])))
            p.setup(*_flow(d, seed + 7 * k, 10.0 ** amp.uniform(-4.0, -2.0)))
            t = 0.0
            for _ in range(c["steps"]):
                t = p.advance(t)
            out.append(torch.stack(p.project(p.state)))
            ts.append(t)
            k += 1
    return {"svor": out, "t": ts}
