"""The work that users of the fractional-step engine have it do, as cases that
can be timed and compared: single Engines in every form (plain FP64, FP64 with
the multigrid projection, FP64 with MacCormack advection, mixed precision),
the diagnostics a run prints, a Batch of uneven grids and a served stream.

A case's pass advances its grids by whole Steps, as a simulation loop does
between two outputs, and reads the state back.  Passes go on from the state
the last one left.

Initial fields: a divergence-free vortex that fits the box's walls plus
uniform noise, made from the seed on the device in binary64.  exact() steps
the same fields in plain torch binary64: the forms that project to a
tolerance are compared with the exact (discrete cosine) projection.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from aeroflux_gb300 import (AF_ADVECTION_MACCORMACK, AF_PRECISION_FP64, AF_PRECISION_MIXED, Config, New)
from aeroflux_gb300.batch import Batch
from aeroflux_gb300.serve import Server

# H = 1/max extent and DT = 0.256 H / amplitude (a CFL number of 0.256, as the
# 64^3, 256^3 and 512^3 configurations have), unless the form says otherwise.
BATCH_DIMS = (32, 48, 64, 96, 128)        # the batched workload's extents
SERVE_DIMS = tuple(range(32, 193, 16))    # the served stream's extents


def listed():
    return [
        # The package's Example: a 16^3 shear layer stepped at 60 sweeps, one
        # Step per call with the state looked at in between (latency).
        dict(name="fp64_16", form="fp64", nx=16, ny=16, nz=16, gsi=60, steps=1, noise=0.01),
        # A small duct-like box of odd extents at the default 24 sweeps.
        dict(name="fp64_odd", form="fp64", nx=97, ny=34, nz=51, gsi=24, steps=4, noise=0.01),
        # The 64^3, default-sweeps configuration that runs for 1000 Steps.
        dict(name="fp64_64", form="fp64", nx=64, ny=64, nz=64, gsi=24, steps=10, noise=0.01),
        # The headline 256^3 configuration, 200 sweeps a projection.
        dict(name="fp64_256", form="fp64", nx=256, ny=256, nz=256, gsi=200, steps=1, noise=0.01),
        # A large ragged grid at the default sweep count.
        dict(name="fp64_ragged", form="fp64", nx=250, ny=171, nz=133, gsi=24, steps=2, noise=0.02),
        # Exact projection with the reference's sweeps, medium size.
        dict(name="multigrid_192", form="multigrid", nx=192, ny=160, nz=128, gsi=24, steps=2, noise=0.01),
        # Higher-order advection, medium size.
        dict(name="maccormack_128", form="maccormack", nx=128, ny=128, nz=128, gsi=24, steps=2, noise=0.01),
        # What a run prints between outputs: max divergence, kinetic energy, CFL.
        dict(name="diagnostics_256", form="diagnostics", nx=256, ny=256, nz=256, gsi=24, steps=0, noise=0.01),
        # A small mixed-precision grid (launches count).
        dict(name="mixed_48", form="mixed", nx=48, ny=32, nz=64, gsi=24, steps=8, noise=0.01),
        # The mixed-precision form at the two benchmark sizes.
        dict(name="mixed_256", form="mixed", nx=256, ny=256, nz=256, gsi=24, steps=8, noise=0.01),
        dict(name="mixed_512", form="mixed", nx=512, ny=512, nz=512, gsi=24, steps=4, noise=0.05),
        # 256 uneven independent grids stepping together.
        dict(name="batch_256", form="batch", grids=256, steps=4, noise=0.01),
    ]


def draw(rng):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    form = rng.choice(["fp64", "fp64", "fp64", "multigrid", "maccormack", "diagnostics", "mixed", "mixed", "mixed",
                       "batch", "batch", "served"])
    if form == "batch":
        return dict(form=form, grids=between(4, 256), steps=rng.randint(1, 4), noise=rng.uniform(0.005, 0.05))
    if form == "served":
        return dict(form=form, requests=between(3, 24), steps=rng.randint(2, 10), noise=rng.uniform(0.005, 0.05))
    if form in ("mixed", "multigrid"):  # extents that coarsen: multiples of 16 in the served range and beyond
        n = [16 * between(2, 18) for _ in range(3)]
    else:
        n = [between(12, 272) for _ in range(3)]
    c = dict(form=form, nx=n[0], ny=n[1], nz=n[2], gsi=24, steps=0, noise=rng.uniform(0.005, 0.05))
    if form != "diagnostics":
        c["steps"] = rng.randint(1, 4)
    if form == "fp64":
        c["gsi"] = between(16, 200)
    return c


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _grid(nx, ny, nz, noise, nu=1e-5, cap=math.inf):
    h = 1.0 / max(nx, ny, nz)
    return dict(nx=nx, ny=ny, nz=nz, h=h, dt=min(0.256 * h, cap), nu=nu, noise=noise)


def _grids(case, seed):
    """The grids of a case, each with the seed of its own noise."""
    if "nx" in case:
        return [dict(_grid(case["nx"], case["ny"], case["nz"], case["noise"]), seed=seed)]
    # Uneven grids: extents by the workload's own distribution, the viscosity
    # log-uniform in [1e-6, 1e-4], DT at half the diffusion limit at most.
    # The mix belongs to the case, the fields to the seed.
    rng, out = random.Random(case.get("grids", case.get("requests"))), []
    for k in range(case.get("grids", case.get("requests"))):
        nx, ny, nz = (rng.choice(BATCH_DIMS if case["form"] == "batch" else SERVE_DIMS) for _ in range(3))
        nu = 10.0 ** rng.uniform(-6.0, -4.0)
        h = 1.0 / max(nx, ny, nz)
        out.append(dict(_grid(nx, ny, nz, case["noise"], nu, min(0.004, 0.5 * h * h / (6.0 * nu))),
                        seed=1009 * seed + k))
    return out


def _fields(g):
    """U, V, W of a grid, padded as the engine lays them out (z, y, x; ghost 1),
    zero outside the faces that carry flow."""
    dev, f64 = _device(), torch.float64
    nx, ny, nz = g["nx"], g["ny"], g["nz"]
    gen = torch.Generator(device=dev)
    gen.manual_seed(g["seed"])

    def centre(n):
        return 2 * math.pi * (torch.arange(n, dtype=f64, device=dev) + 0.5) / n

    def face(n):
        return 2 * math.pi * torch.arange(n + 1, dtype=f64, device=dev) / n

    def noisy(x, y, z, amp):
        a = z[:, None, None] * y[None, :, None] * (amp * x)[None, None, :]
        return a + g["noise"] * (2 * torch.rand(a.shape, dtype=f64, device=dev, generator=gen) - 1)

    u = torch.zeros(nz + 2, ny + 2, nx + 3, dtype=f64, device=dev)
    v = torch.zeros(nz + 2, ny + 3, nx + 2, dtype=f64, device=dev)
    w = torch.zeros(nz + 3, ny + 2, nx + 2, dtype=f64, device=dev)
    u[1:-1, 1:-1, 1:-1] = noisy(face(nx).sin(), centre(ny).cos(), centre(nz).cos(), nx / max(nx, ny))
    v[1:-1, 1:-1, 1:-1] = noisy(centre(nx).cos(), face(ny).sin(), centre(nz).cos(), -ny / max(nx, ny))
    w[1:-1, 1:-1, 1:-1] = noisy(centre(nx).cos(), centre(ny).cos(), face(nz).sin(), 0.0)
    return {"U": u, "V": v, "W": w}


def _config(g, case):
    mixed = case["form"] in ("mixed", "batch", "served")
    return Config(NX=g["nx"], NY=g["ny"], NZ=g["nz"], H=g["h"], DT=g["dt"], Viscosity=g["nu"], Density=1.0,
                  GaussSeidelIters=case.get("gsi", 24), Precision=AF_PRECISION_MIXED if mixed else AF_PRECISION_FP64,
                  DivTol=1e-10 if mixed else 0.0)


def _host(count):
    """A page-locked buffer that a program keeps for reading fields back."""
    return torch.empty(count, dtype=torch.float64, pin_memory=torch.cuda.is_available())


class _State:
    """What a program holds between passes; closes its handle when dropped."""

    def __init__(self, case):
        self.case, self.handle, self.out = case, None, {}

    def __del__(self):
        if self.handle is not None:
            (self.handle.Close if hasattr(self.handle, "Close") else self.handle.close)()


def prepare(case, seed):
    s = _State(case)
    grids = _grids(case, seed)
    if case["form"] == "served":
        # A server that has been up for a while: tuned on requests like these.
        s.handle = Server(16 << 30, max_slots=32, max_round_steps=8, retain=True, max_resident_cells=96 << 20)
        s.requests = [(_config(g, case), g["seed"]) for g in grids]
        for cfg, sd in s.requests:
            s.handle.submit(cfg, 1, seed=sd)
        s.handle.round()
        s.handle.tune(2)
        for r in _drain(s):
            s.handle.release(r["id"])
        return s
    if case["form"] == "batch":
        s.handle = Batch(len(grids))
        s.slots = [s.handle.assign(_config(g, case)) for g in grids]
        s.handle.tune(2)
        for slot, g in zip(s.slots, grids):
            for name, a in _fields(g).items():
                s.handle.upload(slot, name, a.cpu().numpy().ravel())
        s.handle.apply_velocity_bc()
        for name in ("U", "V", "W"):
            s.out[name] = _host(sum(s.handle.field(slot, name).Count for slot in s.slots))
        return s
    s.handle = e = New(_config(grids[0], case))
    if case["form"] == "multigrid":
        e.EnableMultigridSolver()
    if case["form"] == "maccormack":
        e.SetAdvection(AF_ADVECTION_MACCORMACK)
    for name, a in _fields(grids[0]).items():
        e.upload(name, a.cpu().numpy().ravel())
    e.applyVelocityBC()
    if case["form"] != "diagnostics":
        for name in ("U", "V", "W", "P"):
            s.out[name] = _host(getattr(e.Mesh, name).Count)
    return s


def _drain(s):
    while s.handle.stats()["queued"] or s.handle.stats()["resident"]:
        s.handle.round()
    return sorted(s.handle.results(), key=lambda r: r["id"])


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    case, h = s.case, s.handle
    if case["form"] == "diagnostics":
        return [h.MaxDivergence(), h.KineticEnergy(), h.CFL()]
    if case["form"] == "served":
        ids = [h.submit(cfg, case["steps"] + k % 4, seed=sd) for k, (cfg, sd) in enumerate(s.requests)]
        done = _drain(s)
        out = []
        for i, (cfg, _) in zip(ids, s.requests):
            nx, ny, nz = cfg.NX + 2, cfg.NY + 2, cfg.NZ + 2
            for name, n in (("U", (nx + 1) * ny * nz), ("V", nx * (ny + 1) * nz), ("W", nx * ny * (nz + 1))):
                out.append(h.download(i, name, n))
            h.release(i)
        return {"fields": np.concatenate(out), "steps": [int(r["steps"]) for r in done]}
    if case["form"] == "batch":
        h.step(case["steps"])
        for name, buf in s.out.items():
            at = 0
            for slot in s.slots:
                n = h.field(slot, name).Count
                h.download(slot, name, buf[at:at + n].numpy())
                at += n
        return s.out
    h.Step(case["steps"])
    for name, buf in s.out.items():
        h.download(name, buf.numpy())
    return s.out


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    grids, steps = _grids(case, 0), case["steps"]
    cells = sum(g["nx"] * g["ny"] * g["nz"] for g in grids)
    if case["form"] == "diagnostics":
        return {"bytes": 3 * 8 * cells, "flops": 22 * cells}
    # State in and out once: U, V, W and P.
    bytes_ = 2 * 4 * 8 * cells
    sweeps = 6 * 3 * 14          # face velocity, backtrace, interpolation, diffusion
    stages = 2 * (6 + 9)         # divergence and gradient
    if case["form"] == "maccormack":
        sweeps += 6 * 3 * 12
    if case["form"] in ("fp64", "maccormack"):
        solve = 2 * 7 * case["gsi"]
    else:  # about seven V-cycles and four binary64 residuals a Step
        solve = 7 * 80 + 4 * 10
    return {"bytes": bytes_, "flops": cells * steps * (sweeps + stages + solve)}


# ---------------------------------------------------------------------------
# The same Steps in plain torch binary64
# ---------------------------------------------------------------------------
_AXIS = {0: 2, 1: 1, 2: 0}  # x, y, z -> tensor dimension


def _sl(ndim3, dim, s):
    i = [slice(1, -1)] * ndim3
    i[dim] = s
    return tuple(i)


def _velocity_bc(vel):
    for c, a in enumerate(vel):
        d = _AXIS[c]
        for k in (1, a.shape[d] - 2):
            a[_sl(3, d, k)] = 0.0
        done = []
        for ax in range(3):
            t = _AXIS[ax]
            if ax == c:
                continue
            rng = [slice(1, -1)] * 3
            for p in done:
                rng[p] = slice(None)
            for ghost, src in ((0, 1), (a.shape[t] - 1, a.shape[t] - 2)):
                to, fr = list(rng), list(rng)
                to[t], fr[t] = ghost, src
                a[tuple(to)] = -a[tuple(fr)]
            done.append(t)


def _pressure_bc(p):
    for d in (2, 1, 0):
        n = p.shape[d]
        p.select(d, 0).copy_(p.select(d, 1))
        p.select(d, n - 1).copy_(p.select(d, n - 2))


def _face_velocity(vel, c, ax):
    """The velocity along `ax` at the faces of component c that are written."""
    a = vel[ax]
    if c == ax:
        return a[1:-1, 1:-1, 1:-1]
    # The two faces around along ax, and the two cells around the face along c.
    n, m = _AXIS[ax], _AXIS[c]
    cells = [slice(1, -1)] * 3
    out = 0.0
    for k in (0, 1):
        for j in (0, 1):
            i = list(cells)
            i[n] = slice(1 + k, a.shape[n] - 2 + k)
            i[m] = slice(j, a.shape[m] - 1 + j)
            out = out + a[tuple(i)]
    return 0.25 * out


def _sweep(vel, tmp, ax, dt, g, maccormack):
    dim, shift = _AXIS[ax], dt / g["h"]
    lam = g["nu"] * dt / (g["h"] * g["h"])
    for c in range(3):
        a = vel[c]
        n = a.shape[dim]
        rows = a[_sl(3, dim, slice(None))]  # every position along the axis
        shape = [1, 1, 1]
        shape[dim] = -1
        at = torch.arange(1, n - 1, dtype=a.dtype, device=a.device).view(shape)
        move = shift * _face_velocity(vel, c, ax)

        def sample(values, foot):
            foot = foot.clamp(0, n - 1)
            i = foot.long().clamp(max=n - 2)
            t = foot - i
            lo, hi = torch.gather(values, dim, i), torch.gather(values, dim, i + 1)
            return lo + t * (hi - lo), lo, hi

        new, lo, hi = sample(rows, at - move)
        here = rows.narrow(dim, 1, n - 2)
        if maccormack:
            there = rows.clone()
            there.narrow(dim, 1, n - 2).copy_(new)
            back = sample(there, at + move)[0]
            best = new + 0.5 * (here - back)
            new = torch.where((best >= torch.minimum(lo, hi)) & (best <= torch.maximum(lo, hi)), best, new)
        lap = lam * (rows.narrow(dim, 0, n - 2) - 2 * here + rows.narrow(dim, 2, n - 2))
        tmp[c][1:-1, 1:-1, 1:-1] = new + lap
    return tmp, vel


def _cosines(n, f64, dev):
    k, i = torch.arange(n, dtype=f64, device=dev)[:, None], torch.arange(n, dtype=f64, device=dev)[None, :]
    c = torch.cos(math.pi * k * (i + 0.5) / n) * math.sqrt(2.0 / n)
    c[0] *= math.sqrt(0.5)
    return c, 2 - 2 * torch.cos(math.pi * k[:, 0] / n)


def _project(vel, p, g, gsi):
    _velocity_bc(vel)
    u, v, w = vel
    div = ((u[1:-1, 1:-1, 2:-1] - u[1:-1, 1:-1, 1:-2]) + (v[1:-1, 2:-1, 1:-1] - v[1:-1, 1:-2, 1:-1])
           + (w[2:-1, 1:-1, 1:-1] - w[1:-2, 1:-1, 1:-1])) / (g["dt"] * g["h"])
    b = g["h"] * g["h"] * div
    x = p[1:-1, 1:-1, 1:-1]
    if gsi:
        p.zero_()
        z, y, q = (torch.arange(1, n + 1, device=p.device) for n in b.shape)
        red = (z[:, None, None] + y[None, :, None] + q[None, None, :]) % 2 == 0
        for _ in range(gsi):
            for colour in (red, ~red):
                _pressure_bc(p)
                s = (p[1:-1, 1:-1, :-2] + p[1:-1, 1:-1, 2:] + p[1:-1, :-2, 1:-1] + p[1:-1, 2:, 1:-1]
                     + p[:-2, 1:-1, 1:-1] + p[2:, 1:-1, 1:-1])
                x.copy_(torch.where(colour, (s - b) / 6.0, x))
    else:
        bases = [_cosines(n, b.dtype, b.device) for n in b.shape]
        for d, (c, _) in enumerate(bases):
            b = torch.tensordot(c, b, ([1], [d])).movedim(0, d)
        lam = bases[0][1][:, None, None] + bases[1][1][None, :, None] + bases[2][1][None, None, :]
        lam[0, 0, 0] = 1.0
        b = -b / lam
        b[0, 0, 0] = 0.0
        for d, (c, _) in enumerate(bases):
            b = torch.tensordot(c, b, ([0], [d])).movedim(0, d)
        x.copy_(b)
    _pressure_bc(p)
    scale = g["dt"] / g["h"]
    u[1:-1, 1:-1, 1:-1] -= scale * (p[1:-1, 1:-1, 1:] - p[1:-1, 1:-1, :-1])
    v[1:-1, 1:-1, 1:-1] -= scale * (p[1:-1, 1:, 1:-1] - p[1:-1, :-1, 1:-1])
    w[1:-1, 1:-1, 1:-1] -= scale * (p[1:, 1:-1, 1:-1] - p[:-1, 1:-1, 1:-1])
    _velocity_bc(vel)


def _stepped(case, g):
    f = _fields(g)
    vel = [f["U"], f["V"], f["W"]]
    _velocity_bc(vel)
    p = torch.zeros(g["nz"] + 2, g["ny"] + 2, g["nx"] + 2, dtype=torch.float64, device=vel[0].device)
    tmp = [torch.zeros_like(a) for a in vel]
    gsi = case["gsi"] if case["form"] in ("fp64", "maccormack") else 0
    for _ in range(case["steps"]):
        for axes in ((0, 1, 2), (2, 1, 0)):
            for ax in axes:
                _velocity_bc(vel)
                vel, tmp = _sweep(vel, tmp, ax, 0.5 * g["dt"], g, case["form"] == "maccormack")
            _project(vel, p, g, gsi)
    return vel, p


def exact(case, seed):
    if case["form"] == "served":
        return None  # the server makes its own initial fields
    if case["form"] == "diagnostics":
        g = _grids(case, seed)[0]
        vel, _ = _stepped(case, g)
        u, v, w = vel
        div = ((u[1:-1, 1:-1, 2:-1] - u[1:-1, 1:-1, 1:-2]) + (v[1:-1, 2:-1, 1:-1] - v[1:-1, 1:-2, 1:-1])
               + (w[2:-1, 1:-1, 1:-1] - w[1:-2, 1:-1, 1:-1])) / g["h"]
        energy = sum(((0.5 * (a.narrow(d, 1, a.shape[d] - 3) + a.narrow(d, 2, a.shape[d] - 3)))[
            tuple(slice(None) if k == d else slice(1, -1) for k in range(3))] ** 2).sum()
            for d, a in ((2, u), (1, v), (0, w)))
        fastest = max(float(a.abs().max()) for a in vel)
        return [float(div.abs().max()), float(0.5 * energy * g["h"] ** 3), fastest * g["dt"] / g["h"]]
    if case["form"] == "batch":
        got = [_stepped(case, g)[0] for g in _grids(case, seed)]
        return {n: torch.cat([vel[k].reshape(-1) for vel in got]) for k, n in enumerate(("U", "V", "W"))}
    vel, p = _stepped(case, _grids(case, seed)[0])
    out = {n: a.reshape(-1) for n, a in zip(("U", "V", "W"), vel)}
    # P of a projection to a tolerance is known up to a constant only.
    out["P"] = p.reshape(-1) if case["form"] in ("fp64", "maccormack") else None
    return out
