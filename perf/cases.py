"""The work that a user of swb200 has it do, as cases that can be timed and checked.

A case is a dict of plain values.  ``prepare`` makes what a user's program has in hand before the call (a set-up
model with its state, host arrays, ensemble members), ``run`` makes one pass through the public entry points, ``work``
counts what a pass cannot do without and ``exact`` computes the same outputs in 64 bits with plain torch, written from
the model's equations.

kinds
  frames    a device-resident ``Model``: advance ``steps`` steps and read the whole state back (an output frame);
            passes continue the run
  dropin    ``time_integration``: host arrays in, ``steps`` steps, host arrays out
  run_model ``run_model``: keyword arguments in, final fields out
  ensemble  ``run_batched`` over seeded members of uneven size
  gradient  ``adjoint.gradient`` of an eta misfit
"""
from __future__ import annotations

import functools
import json
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "shallowwaters.jl_b200"))

import swb200  # noqa: E402
from swb200 import adjoint, ensemble  # noqa: E402

FORMATS = {"f32": np.float32, "f64": np.float64}

#: The options a case may set, with the values a case that does not name them has.
DEFAULTS = dict(nx=100, L_ratio=2, T="f32", bc="periodic", alpha=2.0, scheme="RK", RKo=4, RKs=3, adv="ArakawaHsu",
                diffusion="Smagorinsky", drag="quadratic", topography="flat", wind="channel", tracer=True, Uadv=1000.0,
                storage="native", steps=100, Ndays=1.0, members=0, checkpoints=0)


def listed():
    return [
        # The README's first call: the 100x50 channel through run_model, one day (about 300 steps) from seeded noise.
        dict(name="run_model_100x50", kind="run_model", nx=100, Ndays=1.0),
        # The smallest calls: a program that looks at a tiny model's state every few steps (coupling, plotting).
        # The reference's default options: ridge, constant diffusion, tracer step once in a few hundred steps.
        dict(name="frames_64x32", kind="frames", nx=64, steps=8, topography="ridge", diffusion="constant", Uadv=0.25),
        # Ordinary research run with the default options and a size that no tile divides.
        dict(name="ridge_1000x500", kind="frames", nx=1000, steps=100, topography="ridge", diffusion="constant",
             Uadv=0.25),
        # The benchmark's workload: the 2048x1024 channel, tracer every step.
        dict(name="channel_2048x1024", kind="frames", nx=2048, steps=200),
        # The largest: a ragged closed basin over a seamount, beyond what L2 holds.
        dict(name="basin_2999x1500", kind="frames", nx=2999, steps=200, bc="nonperiodic", alpha=0.5,
             topography="seamount", wind="double_gyre"),
        # The drop-in call on host arrays: the 512x512 free-slip double gyre over a seamount.
        dict(name="gyre_dropin_512x512", kind="dropin", nx=512, L_ratio=1, steps=200, bc="nonperiodic", alpha=0.0,
             topography="seamount", wind="double_gyre"),
        # Float64, the format of reference runs.
        dict(name="channel_f64_512x256", kind="frames", nx=512, steps=200, T="f64"),
        # The other time schemes a user picks: SSPRK3 in Float32, and SSPRK2 with Sadourny advection in Float64.
        dict(name="ssprk3_500x250", kind="frames", nx=500, steps=200, scheme="SSPRK3", topography="ridge"),
        dict(name="ssprk2_f64_300x300", kind="frames", nx=300, L_ratio=1, steps=200, T="f64", scheme="SSPRK2",
             adv="Sadourny", bc="nonperiodic", alpha=2.0, wind="double_gyre", drag="linear", Uadv=0.25),
        # The 16-bit storage form at the benchmark's size.
        dict(name="bf16_2048x1024", kind="frames", nx=2048, steps=100, storage="bf16"),
        # A batched ensemble of uneven members (64 to 256 columns, both boundary types), three days.
        dict(name="ensemble_48", kind="ensemble", members=48, Ndays=3.0),
        # The gradient of the 512x256 twin experiment's misfit, every state kept.
        dict(name="gradient_f64_512x256", kind="gradient", nx=512, steps=60, T="f64", tracer=False),
    ]


def _rows(nx, L_ratio):
    return int(round(2000e3 / L_ratio / (2000e3 / nx)))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frames"] * 7 + ["dropin", "dropin", "run_model", "ensemble", "gradient", "gradient"])
    bc = rng.choice(["periodic", "nonperiodic"])
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(8, 44), Ndays=rng.choice([1.0, 2.0, 3.0]),
                    storage=rng.choice(["native", "native", "bf16"]))
    c = dict(kind=kind, bc=bc, alpha=rng.choice([0.0, 0.5, 1.0, 2.0]), L_ratio=rng.choice([1, 2, 2, 3]),
             topography=rng.choice(["flat", "ridge", "seamount", "ridges"]),
             wind=rng.choice(["channel", "double_gyre", "shear"]),
             drag=rng.choice(["quadratic", "quadratic", "linear", "none"]),
             diffusion=rng.choice(["Smagorinsky", "constant"]), T=rng.choice(["f32", "f32", "f64"]))
    if kind == "gradient":
        c.update(nx=_log(rng, 64, 500), steps=rng.randint(10, 50), tracer=False,
                 checkpoints=rng.choice([0, 0, rng.randint(4, 9)]), scheme=rng.choice(["RK", "RK", "SSPRK2"]))
        return c
    c["Uadv"] = rng.choice([0.25, 10.0, 1000.0])
    if kind == "run_model":
        c.update(nx=_log(rng, 48, 200), Ndays=rng.choice([0.5, 1.0]))
        return c
    c.update(scheme=rng.choice(["RK", "RK", "RK", "SSPRK2", "SSPRK3", "4SSPRK3"]),
             adv=rng.choice(["ArakawaHsu", "ArakawaHsu", "Sadourny"]))
    c["nx"] = _log(rng, 48, 1400 if c["T"] == "f64" else 2800)
    cells = c["nx"] * _rows(c["nx"], c["L_ratio"])
    c["steps"] = max(8, min(_log(rng, 8, 300), int(4e8 / cells / (2 if c["T"] == "f64" else 1))))
    if c["T"] == "f32" and c["scheme"] == "RK" and c["adv"] == "ArakawaHsu" and rng.random() < 0.3:
        c["storage"] = rng.choice(["bf16", "f16"])
    return c


def _full(case):
    return {**DEFAULTS, **case}


# ------------------------------------------------------------------ set-up through the package

def _kwargs(c):
    return dict(nx=c["nx"], L_ratio=c["L_ratio"], bc=c["bc"], α=c["alpha"], time_scheme=c["scheme"], RKo=c["RKo"],
                RKs=c["RKs"], adv_scheme=c["adv"], diffusion=c["diffusion"], bottom_drag=c["drag"],
                topography=c["topography"], wind_forcing_x=c["wind"], tracer_advection=c["tracer"], Uadv=c["Uadv"],
                Ndays=c["Ndays"])


@functools.lru_cache(maxsize=4)
def _setup(key):
    c = json.loads(key)
    return swb200.model_setup(swb200.Parameter(T=FORMATS[c["T"]], **_kwargs(c)))


def _fields(c, seed):
    """Interior fields at the start: a flow of a few tenths of a metre per second in long waves, eta with the same and
    the benchmark's noise of a centimetre, the tracer a +-1 checkerboard, all rounded to the case's format."""
    nx, ny = c["nx"], _rows(c["nx"], c["L_ratio"])
    nux = nx if c["bc"] == "periodic" else nx - 1
    rng = np.random.default_rng(seed)
    T = FORMATS[c["T"]]

    def waves(h, w, peak):
        x, y = np.arange(w) / nx, (np.arange(h) + 0.5) / ny
        f = np.zeros((h, w))
        for _ in range(3):
            kx, ky = rng.integers(1, 4, size=2)
            ph = rng.uniform(0, 2 * np.pi)
            f += rng.uniform(0.5, 1.0) * peak / 3 * np.outer(np.sin(np.pi * ky * y), np.cos(2 * np.pi * kx * x + ph))
        return f

    u, v = waves(ny, nux, 0.3), waves(ny - 1, nx, 0.2)
    eta = waves(ny, nx, 0.1) + rng.normal(0.0, 0.01, (ny, nx))
    block = max(2, nx // 10)
    i, j = np.arange(nx)[None, :], np.arange(ny)[:, None]
    sst = np.where(((i // block) + (j // block)) % 2 == 0, 1.0, -1.0)
    return tuple(a.astype(T) for a in (u, v, eta, sst))


def _observations(c, seed):
    nx, ny = c["nx"], _rows(c["nx"], c["L_ratio"])
    rng = np.random.default_rng(seed + 7919)
    return (_fields(c, seed)[2] + rng.normal(0.0, 0.02, (ny, nx))).astype(FORMATS[c["T"]])


def prepare(case, seed):
    c = _full(case)
    if c["kind"] == "ensemble":
        members = ensemble.c4_members(c["members"], Ndays=c["Ndays"])     # the benchmark's members, other noise
        for k, m in enumerate(members):
            m.seed = seed * 1000 + k
        return dict(c=c, members=members)
    S = _setup(json.dumps({k: c[k] for k in DEFAULTS}, sort_keys=True))
    u, v, eta, sst = _fields(c, seed)
    state = dict(c=c, S=S)
    if c["kind"] == "run_model":
        state["kw"] = dict(_kwargs(c), u0=u, v0=v, η0=eta, sst0=sst)
        return state
    state["prog"] = swb200.initial_conditions(S.parameters.Tprog, S, u0=u, v0=v, η0=eta, sst0=sst)
    if c["kind"] == "gradient":
        state["obs"] = _observations(c, seed)
    if c["kind"] == "frames":
        state["model"] = swb200.Model(S, storage=c["storage"])
        state["model"].set_state(state["prog"])
    return state


def run(state):
    c = state["c"]
    if c["kind"] == "frames":
        state["model"].run(c["steps"])
        return tuple(state["model"].get_state())
    if c["kind"] == "dropin":
        return tuple(swb200.time_integration(state["prog"], state["S"], nt=c["steps"], storage=c["storage"])[0])
    if c["kind"] == "run_model":
        return tuple(swb200.run_model(FORMATS[c["T"]], **state["kw"]))
    if c["kind"] == "ensemble":
        rows, final = ensemble.run_batched(state["members"], return_states=True, storage=c["storage"])
        order = sorted(final)
        return tuple(np.concatenate([final[k][f].ravel() for k in order]) for f in range(4)) + \
            (np.stack([rows[k] for k in order]),)
    r = adjoint.gradient(state["S"], state["prog"], state["obs"], c["steps"], c["checkpoints"] or c["steps"])
    return r.J, r.u, r.v, r.eta, r.Fx, r.eta_final


# ------------------------------------------------------------------ what a pass cannot do without

def _counts(nx, ny, steps, size, c, uadv_step):
    """Each step reads the state once and writes it once (the tracer on the steps that move it); operations of the
    model's equations per cell: about 115 per right-hand side, 110 for drag and diffusion, 75 for the tracer."""
    sub = {"RK": c["RKo"], "SSPRK2": c["RKs"], "SSPRK3": 4, "4SSPRK3": 4}[c["scheme"]]
    tracer = 1.0 / uadv_step if c["tracer"] else 0.0
    cells = nx * ny * steps
    return {"bytes": cells * size * (6 + 4 * tracer), "flops": cells * (115.0 * sub + 110.0 + 75.0 * tracer)}


def _step_seconds(nx):
    d = 2000e3 / nx
    return d, math.floor(d / math.sqrt(10.0 * 500.0))


def work(case):
    c = _full(case)
    if c["kind"] == "ensemble":
        total = {"bytes": 0.0, "flops": 0.0}
        for m in ensemble.c4_members(c["members"], Ndays=c["Ndays"]):
            nx = m.kwargs["nx"]
            nt = math.ceil(c["Ndays"] * 86400 / _step_seconds(nx)[1])
            w = _counts(nx, _rows(nx, m.kwargs["L_ratio"]), nt, 2 if c["storage"] != "native" else 4, c, 280)
            total = {k: total[k] + w[k] for k in total}
        return total
    nx, ny = c["nx"], _rows(c["nx"], c["L_ratio"])
    d, dt = _step_seconds(nx)
    steps = math.ceil(c["Ndays"] * 86400 / dt) if c["kind"] == "run_model" else c["steps"]
    size = 2 if c["storage"] != "native" else np.dtype(FORMATS[c["T"]]).itemsize
    w = _counts(nx, ny, steps, size, c, max(1, math.floor(d / c["Uadv"] / dt)))
    # forward sweep, and a reverse sweep of twice its operations that reads the states and carries the adjoint
    return {"bytes": 3 * w["bytes"], "flops": 3 * w["flops"]} if c["kind"] == "gradient" else w


# ------------------------------------------------------------------ the same in 64 bits, in plain torch

def _dx(a):
    return a[:, 1:] - a[:, :-1]


def _dy(a):
    return a[1:] - a[:-1]


def _ix(a):
    return 0.5 * (a[:, 1:] + a[:, :-1])


def _iy(a):
    return 0.5 * (a[1:] + a[:-1])


def _ixy(a):
    return _iy(_ix(a))


def _lap(a):
    return a[1:-1, :-2] + a[1:-1, 2:] + a[:-2, 1:-1] + a[2:, 1:-1] - 4 * a[1:-1, 1:-1]


def _root(a):
    """sqrt with derivative 0 at 0."""
    return torch.where(a > 0, torch.sqrt(torch.where(a > 0, a, torch.ones_like(a))), torch.zeros_like(a))


class _Exact:
    """Shallow water on the C-grid in Float64: rows are y, columns are x, u and v carry two halo points and eta one."""

    def __init__(self, c):
        self.c = c
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        nx, Lx, H0, R, omega = c["nx"], 2000e3, 500.0, 6.371e6, 2 * math.pi / 86400
        d, dt = _step_seconds(nx)
        ny = _rows(nx, c["L_ratio"])
        Ly = ny * d
        self.nx, self.ny, self.d, self.dt = nx, ny, d, dt
        self.ep = ep = 1 if c["bc"] == "periodic" else 0
        self.nux = nux = nx if ep else nx - 1
        f0, beta = 2 * omega * math.sin(math.radians(45.0)), 2 * omega / R * math.cos(math.radians(45.0))
        self.fq = self.t(d * (f0 + beta * (d * np.arange(ny + 1) - Ly / 2)))[:, None]
        y = (d * np.arange(1, ny + 1) - d / 2) / Ly - 0.5
        shape = {"channel": np.cos(np.pi * y) ** 2, "shear": np.tanh(2 * np.pi * y),
                 "double_gyre": np.cos(2 * np.pi * y) + 2 * np.sin(np.pi * y)}[c["wind"]]
        self.Fx = self.t(np.tile((d * 0.12 / 1e3 / H0) * shape[:, None], (1, nux)))
        xh, yh = (d * np.arange(0, n + 2) - d / 2 for n in (nx, ny))
        width, high = 300e3, 50.0
        bump = lambda a, at: np.exp(-(a - at) ** 2 / (2 * width ** 2))  # noqa: E731
        flat = np.full((ny + 2, nx + 2), H0)
        self.H = self.t({
            "flat": lambda: flat, "ridge": lambda: flat - high * bump(xh, Lx / 2)[None, :],
            "seamount": lambda: flat - high * np.outer(bump(yh, Ly / 2), bump(xh, Lx / 2)),
            "ridges": lambda: flat - high * sum(bump(xh, at) for at in (
                0.0, 0.99 * Lx / 4, 1.01 * Lx / 2, 0.99 * 3 * Lx / 4, Lx))[None, :]}[c["topography"]]())
        self.slip = 1 - c["alpha"]
        self.cD, self.rD = -d * 1e-5, -d / (300.0 * 86400)
        self.smag, self.nu = -0.15, -500.0 / 30000
        self.nadv = max(1, math.floor(d / c["Uadv"] / dt))
        self.i = 0

    def t(self, a):
        return torch.as_tensor(np.asarray(a, dtype=np.float64), device=self.dev)

    # -- boundaries
    def ghost_uv(self, u, v):
        if self.ep:
            return tuple(torch.cat([a[:, -4:-2], a[:, 2:-2], a[:, 2:4]], 1) for a in (u, v))
        s = self.slip
        return (torch.cat([s * u[3:4], s * u[2:3], u[2:-2], s * u[-3:-2], s * u[-4:-3]], 0),
                torch.cat([s * v[:, 3:4], s * v[:, 2:3], v[:, 2:-2], s * v[:, -3:-2], s * v[:, -4:-3]], 1))

    def ghost_x(self, a):
        if self.ep:
            return torch.cat([a[:, -2:-1], a[:, 1:-1], a[:, 1:2]], 1)
        return torch.cat([a[:, 1:2], a[:, 1:-1], a[:, -2:-1]], 1)

    def ghost_eta(self, e):
        e = self.ghost_x(e)
        return torch.cat([e[1:2], e[1:-1], e[-2:-1]], 0)

    # -- tendencies
    def fluxes(self, u, v, e):
        h, ep = e + self.H, self.ep
        hu, hv = _ix(h), _iy(h)
        n, m = hu.shape
        k, w = hv.shape
        return h, u[1:1 + n, 1 + ep:1 + ep + m] * hu, v[1:1 + k, 1:1 + w] * hv

    def momentum(self, u, v, e):
        nx, ny, ep, nux = self.nx, self.ny, self.ep, self.nux
        h, U, V = self.fluxes(u, v, e)
        hq = _ixy(h)
        n, m = hq.shape
        q = (self.fq + _dx(v)[1:1 + n, 1:1 + m] - _dy(u)[1:1 + n, 1 + ep:1 + ep + m]) / hq
        if self.c["adv"] == "Sadourny":
            s = slice(1 - ep, 1 - ep + nux)
            qhv = _iy(q)[:, s] * _ixy(V)[:, s]
            qhu = _ix(q)[1:ny] * _ixy(U)[1:ny]
        else:
            left = torch.cat([q[:, -1:], q[:, :-1]], 1)     # the first column's left neighbour is the last corner
            a = (q[:-1, :-1] + q[1:, :-1] + q[1:, 1:]) / 12
            b = (q[:-1] + q[1:] + left[1:]) / 12
            g = (q[:-1] + left[:-1] + q[1:]) / 12
            dl = (q[:-1, :-1] + q[1:, :-1] + q[:-1, 1:]) / 12
            s, hi, lo = (slice(k - ep, k - ep + nux) for k in (1, 2, 1))
            qhv = a[:, s] * V[1:, hi] + b[:, s] * V[1:, lo] + g[:, s] * V[:-1, lo] + dl[:, s] * V[:-1, hi]
            qhu = (a[:ny - 1] * U[1:ny, :nx] + b[:ny - 1, 1:] * U[1:ny, 1:1 + nx]
                   + g[1:ny, 1:] * U[2:1 + ny, 1:1 + nx] + dl[1:ny] * U[2:1 + ny, :nx])
        KEu, KEv = _ix(u * u), _iy(v * v)
        p = 0.5 * (KEu[1:3 + ny, ep:ep + nx + 2] + KEv[:ny + 2, 1:3 + nx]) + 10.0 * e
        du = qhv - _dx(p)[1:1 + ny, 1 - ep:1 - ep + nux] + self.Fx
        dv = -(qhu + _dy(p)[1:ny, 1:1 + nx])
        return F.pad(du, (2, 2, 2, 2)), F.pad(dv, (2, 2, 2, 2)), (U, V)

    def continuity(self, UV):
        U, V = UV
        return F.pad(-(_dx(U)[1:1 + self.ny] + _dy(V)[:, 1:1 + self.nx]), (1, 1, 1, 1))

    # -- drag and diffusion
    def tail(self, u, v, e):
        nx, ny, ep, nux = self.nx, self.ny, self.ep, self.nux
        Bu, Bv = 0.0, 0.0
        su, sv = u[2:2 + ny, 2:2 + nux], v[2:1 + ny, 2:2 + nx]
        if self.c["drag"] == "quadratic":
            h = e + self.H
            k = _root(_ix(u * u)[1:3 + ny, ep:ep + nx + 2] + _iy(v * v)[:ny + 2, 1:3 + nx])
            s = slice(1 - ep, 1 - ep + nux)
            Bu = self.cD * _ix(k)[1:1 + ny, s] * su / _ix(h)[1:1 + ny, s]
            Bv = self.cD * _iy(k)[1:ny, 1:1 + nx] * sv / _iy(h)[1:ny, 1:1 + nx]
        elif self.c["drag"] == "linear":
            Bu, Bv = self.rD * su, self.rD * sv
        Lu, Lv = _lap(u), _lap(v)
        ax, ay, bx, by = _dx(Lu), _dy(Lu), _dx(Lv), _dy(Lv)
        ay = ay[:, ep:ep + nx + 1]
        if self.c["diffusion"] == "Smagorinsky":
            shear = _dy(u)[:, ep:ep + nx + 3] + _dx(v)
            div = _dx(u)[1:3 + ny, ep:ep + nx + 2] + _dy(v)[:ny + 2, 1:3 + nx]
            nu = self.smag * _root(_ixy(shear * shear) + div * div)
            nuq = _ixy(nu)
            ax, ay, bx, by = nu[:, 1 - ep:2 - ep + nux] * ax, nuq * ay, nuq * bx, nu[1:1 + ny] * by
        else:
            ax, ay, bx, by = (self.nu * a for a in (ax, ay, bx, by))
        k = self.dt / self.d
        u = u + F.pad(k * (Bu + _dx(ax)[1:1 + ny] + _dy(ay)[:, 1 - ep:1 - ep + nux]), (2, 2, 2, 2))
        v = v + F.pad(k * (Bv + _dx(bx)[1:ny] + _dy(by)[:, 1:1 + nx]), (2, 2, 2, 2))
        return self.ghost_uv(u, v)

    # -- semi-Lagrangian tracer
    def at(self, f, x, y, x1, x2, y1, y2):
        """f at the departure points (cell + displacement), bilinear; x1, x2, y1, y2: f's halo columns and rows."""
        nf, mf = f.shape
        xi, yi = torch.floor(x), torch.floor(y)
        i = xi.long() + torch.arange(1, x.shape[1] + 1, device=self.dev)[None, :] + x1
        j = yi.long() + torch.arange(1, x.shape[0] + 1, device=self.dev)[:, None] + y1
        x, y = x - xi, y - yi
        if self.ep:
            n = mf - x1 - x2
            i = torch.where(i < 1 + x1, i + n, torch.where(i > mf - 1, i - n, i))
        else:
            x = torch.where(i < 1 + x1, torch.zeros_like(x), torch.where(i > mf - 1, torch.ones_like(x), x))
            i = i.clamp(1 + x1, mf - 1)
        y = torch.where(j < 1 + y1, torch.zeros_like(y), torch.where(j > nf - 1, torch.ones_like(y), y))
        j = j.clamp(1 + y1, nf - 1)
        i, j = i - 1, j - 1
        return (f[j, i] * (1 - x) * (1 - y) + f[j, i + 1] * x * (1 - y) + f[j + 1, i] * (1 - x) * y
                + f[j + 1, i + 1] * x * y)

    def tracer(self, u, v, s):
        nx, ny, ep = self.nx, self.ny, self.ep
        if (self.i + self.nadv // 2) % self.nadv == 0:
            self.um, self.vm = u, v
        if self.i % self.nadv:
            return s
        cx = cy = self.nadv * self.dt / self.d
        x = -0.5 * cx * _ix(u)[2:2 + ny, 1 + ep:1 + ep + nx]
        y = -0.5 * cy * _iy(v)[1:1 + ny, 2:2 + nx]
        um = self.at(_ix(self.um), x, y, 1 + ep, 1, 2, 2)
        vm = self.at(_iy(self.vm), x, y, 2, 2, 1, 1)
        return self.ghost_x(F.pad(self.at(s, -cx * um, -cy * vm, 1, 1, 0, 0), (1, 1)))

    # -- one time step
    def step(self, u, v, e, s):
        c, k = self.c, self.dt / self.d
        self.i += 1
        (u, v), e = self.ghost_uv(u, v), self.ghost_eta(e)
        scheme = c["scheme"]
        if scheme == "RK":
            a, b = {2: ([1 / 2, 1 / 2], [1.0]), 3: ([1 / 4, 0.0, 3 / 4], [1 / 3, 2 / 3]),
                    4: ([1 / 6, 1 / 3, 1 / 3, 1 / 6], [0.5, 0.5, 1.0])}[c["RKo"]]
            un, vn, en = u, v, e
            u1, v1, e1 = u, v, e
            for r in range(c["RKo"]):
                du, dv, UV = self.momentum(u1, v1, e1)
                de = self.continuity(UV)
                un, vn, en = un + a[r] * k * du, vn + a[r] * k * dv, en + a[r] * k * de
                if r + 1 < c["RKo"]:
                    u1, v1 = self.ghost_uv(u + b[r] * k * du, v + b[r] * k * dv)
                    e1 = self.ghost_eta(e + b[r] * k * de)
        else:
            def sub(u1, v1, e1, mix):
                du, dv, _ = self.momentum(u1, v1, e1)
                nu, nv = self.ghost_uv(mix(0, u1, du), mix(1, v1, dv))
                return nu, nv, mix(2, e1, self.continuity(self.fluxes(nu, nv, e1)[1:]))

            un, vn, en = u, v, e
            if scheme == "SSPRK2":
                n = c["RKs"]
                for r in range(n):
                    un, vn, en = sub(un, vn, self.ghost_eta(en), lambda f, x, d: x + k / (n - 1) * d)
                un, vn, en = (x / n + (n - 1) / n * y for x, y in ((u, un), (v, vn), (e, en)))
            elif scheme == "SSPRK3":                      # four sub-stages, the last but one mixes in the start
                u0, v0, e0 = u, v, e
                for r in (2, 3, 4, 5):
                    if r == 4:
                        z = (u0, v0, e0)
                        mix = lambda f, x, d: x / 3 + 2 / 3 * z[f] + k / 6 * d  # noqa: E731
                    else:
                        mix = lambda f, x, d: x + k / 2 * d  # noqa: E731
                    un, vn, en = sub(un, vn, self.ghost_eta(en), mix)
            else:
                for r in range(4):
                    if r:
                        (un, vn), en = self.ghost_uv(un, vn), self.ghost_eta(en)
                    un, vn, en = sub(un, vn, en, lambda f, x, d: x + 0.5 * k * d)
                    if r == 2:
                        un, vn, en = (2 / 3 * x + y / 3 for x, y in ((u, un), (v, vn), (e, en)))
        (un, vn), en = self.ghost_uv(un, vn), self.ghost_eta(en)
        un, vn = self.tail(un, vn, en)
        if c["tracer"]:
            s = self.tracer(un, vn, s)
        return un, vn, en, s

    def start(self, seed):
        u, v, e, s = (self.t(a) for a in _fields(self.c, seed))
        u, v = self.ghost_uv(F.pad(u, (2, 2, 2, 2)), F.pad(v, (2, 2, 2, 2)))
        self.um, self.vm = torch.zeros_like(u), torch.zeros_like(v)
        return u, v, self.ghost_eta(F.pad(e, (1, 1, 1, 1))), self.ghost_x(F.pad(s, (1, 1)))


def exact(case, seed):
    c = _full(case)
    if c["kind"] == "ensemble":        # tens of thousands of member steps: minutes
        return None
    m = _Exact(c)
    steps = math.ceil(c["Ndays"] * 86400 / m.dt) if c["kind"] == "run_model" else c["steps"]
    state = m.start(seed)
    if c["kind"] == "gradient":
        u, v, e = (a.clone().requires_grad_() for a in state[:3])
        m.Fx.requires_grad_()
        x = (u, v, e, state[3])
        for _ in range(steps):
            x = m.step(*x)
        J = ((x[2][1:-1, 1:-1] - m.t(_observations(c, seed))) ** 2).sum()
        g = torch.autograd.grad(J, (u, v, e, m.Fx))
        return [J.item()] + [a.cpu().numpy() for a in g] + [x[2].detach().cpu().numpy()]
    with torch.no_grad():
        for _ in range(steps):
            state = m.step(*state)
    out = [a.cpu().numpy() for a in state]
    if c["kind"] == "frames":
        return out
    cut = lambda a, x, y: a[y:a.shape[0] - y, x:a.shape[1] - x]  # noqa: E731
    return [np.ascontiguousarray(cut(a, *h)) for a, h in zip(out, ((2, 2), (2, 2), (1, 1), (1, 0)))]
