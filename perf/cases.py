"""Performance cases of picsar_b200: the calls a simulation program makes.

Each case is a plain dict; ``prepare`` builds the simulation or the arrays a
program holds before the call, ``run`` is one pass through the public entry
points with the outputs such a program reads, ``exact`` is the same result in
64 bits from plain torch on periodic grids (no code of this package).

Kinds:
  tiled         ``TiledSim.step`` and the read-out of fields and particles
  module_tiled  ``PicsarModule(engine="tiled")``: steps, then module arrays
  module        ``PicsarModule`` on PICSAR's own FP64 arrays
  module2d      ``PicsarModule2D`` (x-z)
  ensemble      ``Ensemble.step`` over uneven jobs
  routines      the separate Forthon routines on a caller's arrays
"""
from __future__ import annotations

import math
import random
from dataclasses import replace

import numpy as np
import torch

from picsar_b200 import picsar as P
from picsar_b200.ensemble import Ensemble, ensemble_jobs
from picsar_b200.init import thermal_plasma, two_stream_ramp
from picsar_b200.tiled import TiledConfig, TiledSim

EB = ("ex", "ey", "ez", "bx", "by", "bz")
J3 = ("jx", "jy", "jz")
COLS = ("x", "y", "z", "ux", "uy", "uz")
G = 3                       # guard cells of the PICSAR-layout arrays


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _tiled(n, ppc, order, precision, acc, steps, sigma=0.01, pusher=0, drift=0.0, lanes=True):
    return {"kind": "tiled", "nx": n[0], "ny": n[1], "nz": n[2], "ppc": ppc, "order": order,
            "precision": precision, "acc": acc, "steps": steps, "sigma": sigma,
            "pusher": pusher, "drift": drift, "lanes": lanes}


def _module(kind, n, ppc, order, steps, sigma=0.01, pusher=0, norder=2, shuffle=False, dx=1.0,
            dz=1.0):
    return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "ppc": ppc, "order": order,
            "steps": steps, "sigma": sigma, "pusher": pusher, "norder": norder,
            "shuffle": shuffle, "dx": dx, "dz": dz}


def listed():
    return [
        # the benchmark's large thermal plasma: one sort period of a production
        # run on a full GPU, then a dump of fields and particles
        dict(_tiled((256, 256, 256), 8, 3, "fp32", 1, 20), name="tiled-large-o3"),
        # the medium plasma with the engine's default settings (two-word
        # current accumulator)
        dict(_tiled((128, 128, 64), 8, 3, "fp32", 2, 20), name="tiled-default-o3"),
        # counter-streaming beams on a density ramp: many particles change
        # cell every step and the tiles are uneven
        dict(_tiled((256, 96, 96), 16, 2, "fp32", 1, 20, sigma=0.005, drift=0.2, lanes=False),
             name="tiled-beams-o2"),
        # the small order-1 box of the tests and decks: launches and latency
        dict(_tiled((32, 32, 32), 8, 1, "fp32", 2, 20), name="tiled-small-o1"),
        # the FP64 engine on the medium plasma
        dict(_tiled((128, 128, 64), 8, 3, "fp64", 3, 20), name="tiled-fp64-o3"),
        # a Forthon-style driver on the tiled engine that reads every module
        # array each few steps; ragged sizes, order 2, Vay
        _module("module_tiled", (72, 60, 84), 6, 2, 5, sigma=0.02, pusher=1)
        | {"name": "module-tiled-o2"},
        # a parameter scan: uneven independent jobs stepped together
        {"name": "ensemble", "kind": "ensemble", "jobs": 24, "lo": 16, "hi": 64, "steps": 20,
         "mix": 2024},
        # the drop-in FP64 module on PICSAR's arrays at the medium size
        _module("module", (128, 128, 64), 8, 3, 1) | {"name": "module-o3"},
        # ... its smallest use: a test or deck box, all latency
        _module("module", (16, 16, 16), 4, 1, 1, sigma=0.05) | {"name": "module-small-o1"},
        # ... odd sizes, particles in no order, Vay, order-4 FDTD, cells that
        # are not cubes
        _module("module", (75, 53, 61), 5, 2, 1, sigma=0.05, pusher=1, norder=4, shuffle=True,
                dx=0.8, dz=1.25) | {"name": "module-odd-o2"},
        # the 2D x-z loop
        _module("module2d", (512, 1, 384), 20, 2, 1, sigma=0.05) | {"name": "module-2d-o2"},
        # a code that calls the separate gather and deposition routines on its
        # own particles (in no order), full-order shapes
        {"name": "routines-o3", "kind": "routines", "nx": 96, "ny": 80, "nz": 64, "ppc": 4,
         "order": 3, "lower": False, "shuffle": True, "sigma": 0.05},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(("tiled", "tiled", "tiled", "module", "module", "module_tiled",
                       "module2d", "ensemble", "routines"))
    sigma = round(math.exp(rng.uniform(math.log(0.002), math.log(0.08))), 4)
    n = tuple(_log(rng, 16, 160) for _ in range(3))
    order = rng.randint(1, 3)
    pusher = rng.randint(0, 1)
    if kind == "tiled":
        precision = rng.choice(("fp32", "fp32", "fp64"))
        ppc = _log(rng, 1, 16)
        drift = round(rng.uniform(0.05, 0.25), 2) if rng.random() < 0.25 else 0.0
        acc = 3 if precision == "fp64" else rng.choice((1, 2))
        return _tiled(n, ppc, order, precision, acc, rng.randint(8, 24), sigma, pusher, drift,
                      rng.random() < 0.7)
    if kind == "ensemble":
        lo = rng.randint(16, 32)
        return {"kind": kind, "jobs": rng.randint(2, 24), "lo": lo,
                "hi": lo + rng.randint(8, 40), "steps": rng.randint(8, 24),
                "mix": rng.randint(1, 10 ** 6)}
    if kind == "module2d":
        return _module(kind, (_log(rng, 24, 700), 1, _log(rng, 24, 700)), _log(rng, 1, 20), order,
                       1, sigma, pusher)
    n = tuple(min(v, 112) for v in n)
    ppc = _log(rng, 1, 8)
    if kind == "routines":
        return {"kind": kind, "nx": n[0], "ny": n[1], "nz": n[2], "ppc": ppc, "order": order,
                "lower": rng.random() < 0.5, "shuffle": rng.random() < 0.5, "sigma": sigma}
    if kind == "module_tiled":
        return _module(kind, n, ppc, order, rng.randint(1, 6), sigma, pusher)
    return _module(kind, n, ppc, order, rng.randint(1, 2), sigma, pusher, rng.choice((2, 2, 4)),
                   rng.random() < 0.5, round(rng.uniform(0.7, 1.3), 2),
                   round(rng.uniform(0.7, 1.3), 2))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _n(c):
    return (c["nx"], c["ny"], c["nz"])


def _d(c):
    return (c.get("dx", 1.0), 1.0, c.get("dz", 1.0))


def _plasma(c, seed, device="cuda"):
    if c.get("drift"):
        return two_stream_ramp(_n(c), c["ppc"], c["drift"], c["sigma"], seed=seed,
                               ramp_cells=max(1, c["nx"] // 2), device=device)
    return thermal_plasma(_n(c), c["ppc"], c["sigma"], seed=seed, d=_d(c), device=device,
                          shuffle=bool(c.get("shuffle")))


def _waves(n, seed, order=3, device="cuda"):
    """Six periodic fields [i, j, k]: a uniform magnetic field along z plus a
    few long waves per component (weak ones at order 1, whose gather jumps
    from cell to cell)."""
    top = 0.001 if order == 1 else 0.02
    rng = np.random.default_rng(seed)
    ax = [2 * math.pi * torch.arange(v, device=device, dtype=torch.float64) / v for v in n]
    out = []
    for q in range(6):
        f = torch.zeros(n, device=device, dtype=torch.float64)
        for _ in range(3):
            m = [int(v) for v in rng.integers(-3, 4, size=3)]
            ph, amp = float(rng.uniform(0, 2 * math.pi)), top * float(rng.uniform(0.5, 1.0))
            f += amp * torch.sin(m[0] * ax[0][:, None, None] + m[1] * ax[1][None, :, None] +
                                 m[2] * ax[2][None, None, :] + ph)
        out.append(f + 0.5 if q == 5 else f)
    return out


def _guarded(f, g=G):
    """Periodic array [i, j, k] as PICSAR's guarded column-major grid (an axis
    of one cell is the absent y axis of x-z grids)."""
    idx = [torch.remainder(torch.arange(-g, v + g + 1, device=f.device), v) if v > 1
           else torch.zeros(1, dtype=torch.int64, device=f.device) for v in f.shape]
    out = f[idx[0]][:, idx[1]][:, :, idx[2]]
    if f.shape[1] == 1:
        out = out[:, 0]
    back = tuple(reversed(range(out.dim())))
    return out.permute(back).contiguous().permute(back)


def _specs(c, seed):
    """The jobs of an ensemble: their sizes from the case, their initial
    states from the seed."""
    jobs = ensemble_jobs(c["jobs"], seed=c["mix"], steps=c["steps"], cells=(c["lo"], c["hi"]))
    return [replace(j, seed=seed * 1000 + i) for i, j in enumerate(jobs)]


def _by_order(items, order_of):
    """{shape order: items of that order, in their order}."""
    out = {}
    for it in sorted(items, key=order_of):           # the ensemble's packed order
        out.setdefault(order_of(it), []).append(it)
    return out


def _starts(specs):
    """Per axis: the jobs' start positions and the period of each."""
    sts = [sp.initial_state() for sp in specs]
    return [(torch.cat([getattr(st, a) for st in sts]),
             torch.cat([torch.full_like(st.x, float(sp.n[q])) for sp, st in zip(specs, sts)]))
            for q, a in enumerate("xyz")]


def _moved(a, start, period):
    """Displacement from the start by the nearest periodic image (what a
    diffusion diagnostic takes; it does not jump at the box's edge)."""
    m = a - start
    return m - period * torch.round(m / period)


def _add(m, c, seed):
    st = _plasma(c, seed)
    if c["kind"] == "module2d":
        st.y.zero_()
    m.add_species("electron", -1.0, 1.0, st.x, st.y, st.z, st.ux, st.uy, st.uz, st.w)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "tiled":
        # beams cross a tile in a few steps: sorted every 5, as the autotuner
        # chooses for them
        cfg = TiledConfig(acc=c["acc"] if c["precision"] == "fp32" else 2,
                          select_lanes=bool(c["lanes"]),
                          sort_interval=5 if c["drift"] else 20)
        sim = TiledSim(_n(c), order=c["order"], pusher=c["pusher"], precision=c["precision"],
                       config=cfg, track_ids=True)
        for name, f in zip(EB, _waves(_n(c), seed, c["order"])):
            sim.import_field(name, _guarded(f), G)
        st = _plasma(c, seed)
        sim.load_state(st)
        return c, sim, [(a, float(v)) for a, v in zip((st.x, st.y, st.z), _n(c))]
    if kind == "ensemble":
        specs = _specs(c, seed)
        ens = Ensemble(specs, track_ids=True)
        return c, ens, {o: _starts(v) for o, v in _by_order(specs, lambda t: t.order).items()}
    if kind == "routines":
        st = _plasma(c, seed)
        z = lambda: torch.zeros_like(st.x)
        gi = 1.0 / torch.sqrt(1.0 + st.ux ** 2 + st.uy ** 2 + st.uz ** 2)
        F = _waves(_n(c), seed, c["order"])
        return c, {"st": st, "gi": gi, "grids": [_guarded(f, 4) for f in F],
                   "part": [z() for _ in EB], "j": [P.grid_zeros(*_n(c), 4) for _ in J3],
                   "err": torch.zeros(1, dtype=torch.int32, device="cuda")}
    if kind == "module2d":
        m = P.PicsarModule2D(c["nx"], c["nz"], nguards=G, nox=c["order"],
                             particle_pusher=c["pusher"])
    else:
        d = _d(c)
        m = P.PicsarModule(*_n(c), nguards=G, nox=c["order"], particle_pusher=c["pusher"],
                           dx=d[0], dy=d[1], dz=d[2], dtcoef=0.8 if c["norder"] > 2 else 0.95,
                           engine="tiled" if kind == "module_tiled" else "plain")
        m.norderx = m.nordery = m.norderz = c["norder"]
    for name, f in zip(EB, _waves(_n(c), seed, c["order"])):
        getattr(m, name).copy_(_guarded(f))
    _add(m, c, seed)
    return c, m


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    c, s = state[:2]
    kind = c["kind"]
    if kind == "tiled":
        s.step(c["steps"])
        out = {name: s.export_field(name, G) for name in EB}
        p = s.particles()
        out.update((k, p[k]) for k in COLS[3:])
        out.update((k, _moved(p[k], *b)) for k, b in zip(COLS[:3], state[2]))
        return out
    if kind == "ensemble":
        s.step(c["steps"])
        out = {}
        for o, sims in _by_order([sim for _, sim in s.sims()], lambda t: t.order).items():
            r = {name: torch.cat([sim.export_field(name, G).permute(2, 1, 0).reshape(-1)
                                  for sim in sims]) for name in EB}
            ps = [sim.particles() for sim in sims]
            r.update((k, torch.cat([p[k] for p in ps])) for k in COLS)
            r.update((k, _moved(r[k], *b)) for k, b in zip(COLS[:3], state[2][o]))
            out["order%d" % o] = r
        return out
    if kind == "routines":
        st, (nx, ny, nz), o = s["st"], _n(c), c["order"]
        for a in s["part"] + s["j"]:
            a.zero_()
        P.geteb3d_energy_conserving(st.np, st.x, st.y, st.z, *s["part"], 0.0, 0.0, 0.0, 1.0, 1.0,
                                    1.0, nx, ny, nz, 4, 4, 4, o, o, o, *s["grids"], False,
                                    c["lower"], 64, 0)
        P.depose_jxjyjz(*s["j"], st.np, st.x, st.y, st.z, st.ux, st.uy, st.uz, s["gi"], st.w,
                        -1.0, 0.0, 0.0, 0.0, 0.5, 1.0, 1.0, 1.0, nx, ny, nz, 4, 4, 4, o, o, o,
                        err_flag=s["err"])
        return dict(zip(EB + J3, s["part"] + s["j"]))
    s.step(c["steps"])
    sp = s.species[0]
    out = {name: getattr(s, name) for name in EB + J3}
    out.update((k, getattr(sp, "part_" + k)) for k in COLS)
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _flops(order, dims=3):
    """Floating-point operations of one particle-step, tensor-product gather
    and the no-node-change Esirkepov box (as bench.py counts them)."""
    n, s = order + 1, order
    shape = {1: (1, 0), 2: (8, 2), 3: (15, 9)}[order]
    if dims == 2:
        pairs = [(s, n), (n, n), (n, s), (n, s), (s, s), (s, n)]
        return (2 * sum(shape) + sum(2 * (a * b + b) for a, b in pairs) + 76 + 10 +
                4 * shape[0] + 12 * n * n)
    comps = [(s, n, n), (n, s, n), (n, n, s), (n, s, s), (s, n, s), (s, s, n)]
    gather = sum(2 * (a * b * c + b * c + c) for a, b, c in comps)
    deposit = 3 * ((2 * n - 3) + n + 5 * n + 4 * n * n + 2 * n * n * (n - 1))
    return 3 * sum(shape) + gather + 76 + 15 + 6 * shape[0] + deposit + 11


def _step_work(cells, np_, order, r, steps, dims=3):
    # per step: x, u read and written, the weight read; E, B read and written,
    # J written and read
    pb = (2 * (dims + 3) + 1) * r
    return {"bytes": steps * (np_ * pb + cells * 18 * r),
            "flops": steps * (np_ * _flops(order, dims) + cells * 81)}


def _particles(c):
    if c.get("drift"):
        dens = np.clip((np.arange(c["nx"]) + 0.5) / max(1, c["nx"] // 2), None, 1.0)
        return int(np.round(dens * c["ppc"]).sum()) * c["ny"] * c["nz"]
    return c["nx"] * c["ny"] * c["nz"] * c["ppc"]


def work(case):
    c, kind = case, case["kind"]
    if kind == "ensemble":
        tot = {"bytes": 0.0, "flops": 0.0}
        for sp in _specs(c, 1):
            w = _step_work(sp.cells, sp.particles, sp.order, 4, c["steps"])
            for k in tot:
                tot[k] += w[k]
            tot["bytes"] += 48 * sp.cells + 48 * sp.particles
        return tot
    np_, cells = _particles(c), c["nx"] * c["ny"] * c["nz"]
    if kind == "routines":
        # x, u, gamma, w read; six fields per particle and J written; E, B read
        return {"bytes": np_ * (8 + 6) * 8 + cells * 9 * 8,
                "flops": np_ * (_flops(c["order"]) - 102)}
    fp32 = kind == "tiled" and c["precision"] == "fp32"
    w = _step_work(cells, np_, c["order"], 4 if fp32 else 8, c["steps"],
                   2 if kind == "module2d" else 3)
    if kind in ("tiled", "module_tiled"):       # the FP64 read-out
        w["bytes"] += 48 * cells + 48 * np_
    return w


def tolerance(case):
    c = case
    if c["kind"] == "ensemble" or (c["kind"] == "tiled" and c["precision"] == "fp32"):
        # FP32 fields, offsets and momenta after the steps, about four times
        # the distance from 64 bits.  At order 1 the staggered shape is a
        # step: a particle within rounding of a cell edge takes the next
        # cell's field.  At order 2 the beams' momenta lose digits against
        # their drift.
        order = 1 if c["kind"] == "ensemble" else c["order"]
        return {"rel": {1: 2e-3, 2: 1e-3, 3: 4e-5}[order], "max": 0.9}
    # FP64 sums in another order, through up to 24 steps; slow particles'
    # currents lose digits (old minus new position)
    return {"rel": 1e-11, "max": 1e-9}


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _spline(deg, xi):
    """B-spline weights of degree 1..3: the support points' values at in-cell
    variable xi (degree 2: distance to the nearest point)."""
    if deg == 0:
        return [torch.ones_like(xi)]
    if deg == 1:
        return [1.0 - xi, xi]
    if deg == 2:
        return [0.5 * (0.5 - xi) ** 2, 0.75 - xi ** 2, 0.5 * (0.5 + xi) ** 2]
    ox = 1.0 - xi
    return [ox ** 3 / 6.0, 2.0 / 3.0 - xi ** 2 * (1.0 - xi / 2.0),
            2.0 / 3.0 - ox ** 2 * (1.0 - ox / 2.0), xi ** 3 / 6.0]


def _shape(deg, x):
    """(first point, weights) of degree deg around x on the integers."""
    if deg in (0, 2):
        i = torch.floor(x + 0.5)
        return (i - deg // 2).long(), _spline(deg, x - i)
    i = torch.floor(x)
    return (i - deg // 2).long(), _spline(deg, x - i)


def _axis(n, first, count):
    return [torch.remainder(first + t, n) for t in range(count)]


def _gather(fields, pos, order, lower):
    n = fields[0].shape
    node = [_shape(order, p) for p in pos]
    stag = [_shape(order - 1 if lower else order, p - 0.5) for p in pos]
    where = ("sNN", "NsN", "NNs", "Nss", "sNs", "ssN")
    out = []
    for f, code in zip(fields, where):
        sh = [stag[a] if code[a] == "s" else node[a] for a in range(3)]
        if n[1] == 1:
            sh[1] = (torch.zeros_like(node[0][0]), [torch.ones_like(pos[0])])
        ix = [_axis(n[a], sh[a][0], len(sh[a][1])) for a in range(3)]
        flat, val = f.reshape(-1), torch.zeros_like(pos[0])
        for i, wi in zip(ix[0], sh[0][1]):
            for j, wj in zip(ix[1], sh[1][1]):
                for k, wk in zip(ix[2], sh[2][1]):
                    val += wi * wj * wk * flat[(i * n[1] + j) * n[2] + k]
        out.append(val)
    return out


def _boris(u, eb, dt):
    h = -0.5 * dt
    u = [a + h * e for a, e in zip(u, eb[:3])]
    gi = 1.0 / torch.sqrt(1.0 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    t = [gi * b * h for b in eb[3:]]
    s = [2.0 * a / (1.0 + t[0] ** 2 + t[1] ** 2 + t[2] ** 2) for a in t]
    cross = lambda a, b: [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2],
                          a[0] * b[1] - a[1] * b[0]]
    up = [a + b for a, b in zip(u, cross(u, t))]
    u = [a + b + h * e for a, b, e in zip(u, cross(up, s), eb[:3])]
    return u, 1.0 / torch.sqrt(1.0 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)


def _vay(u, eb, dt):
    q = -dt
    gi = 1.0 / torch.sqrt(1.0 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    tau = [0.5 * q * b for b in eb[3:]]
    t2 = tau[0] ** 2 + tau[1] ** 2 + tau[2] ** 2
    cross = lambda a, b: [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2],
                          a[0] * b[1] - a[1] * b[0]]
    up = [a + q * e + b * gi for a, e, b in zip(u, eb[:3], cross(u, tau))]
    us = up[0] * tau[0] + up[1] * tau[1] + up[2] * tau[2]
    sg = 1.0 + up[0] ** 2 + up[1] ** 2 + up[2] ** 2 - t2
    gi2 = 2.0 / (sg + torch.sqrt(sg ** 2 + 4.0 * (t2 + us ** 2)))
    gi = torch.sqrt(gi2)
    t = [a * gi for a in tau]
    s = 1.0 / (1.0 + t2 * gi2)
    tu = t[0] * up[0] + t[1] * up[1] + t[2] * up[2]
    return [s * (a + b * tu + x) for a, b, x in zip(up, t, cross(up, t))], gi


def _box(order, xn, xo, const=None):
    """First point, and new / old shapes of one axis on their common box of
    order + 2 points."""
    (i0, s0), (i1, s1) = _shape(order, xn), _shape(order, xo)
    if const is not None and order == 3:
        # the reference's 2-D cubic shape has single-precision constants
        fix = [const[0] * 6.0, None, None, const[0] * 6.0]
        for s in (s0, s1):
            for t in (0, 3):
                s[t] = s[t] * fix[t]
            for t in (1, 2):
                s[t] = s[t] - 2.0 / 3.0 + const[1]
    b = torch.minimum(i0, i1)
    d0, d1 = i0 - b, i1 - b
    z = torch.zeros_like(xn)

    def spread(s, d):
        out = []
        for r in range(order + 2):
            a = s[r] if r <= order else z
            p = s[r - 1] if r >= 1 else z
            out.append(torch.where(d == 0, a, p))
        return out
    return b, spread(s0, d0), spread(s1, d1)


def _deposit(n, new, old, w, d, dt, order, vy=None):
    """Esirkepov currents [i, j, k] of particles of charge -1 (positions in
    cells); n[1] == 1: the x-z form, whose Jy is the transverse current."""
    two = n[1] == 1
    const = (float(np.float32(1) / np.float32(6)), float(np.float32(2) / np.float32(3)))
    third = float(np.float32(1) / np.float32(3)) if two else 1.0 / 3.0
    M = order + 2
    J = [torch.zeros(n[0] * n[1] * n[2], dtype=torch.float64, device=w.device) for _ in range(3)]
    bx, x0, x1 = _box(order, new[0], old[0], const if two else None)
    bz, z0, z1 = _box(order, new[2], old[2], const if two else None)
    ix, iz = _axis(n[0], bx, M), _axis(n[2], bz, M)
    dx_, dz_ = [b - a for a, b in zip(x0, x1)], [b - a for a, b in zip(z0, z1)]
    cum = lambda v: [sum(v[:t + 1]) for t in range(M - 1)]
    if two:
        cx, cz = -w / (dt * d[2]), -w / (dt * d[0])
        for k in range(M):
            for i in range(M):
                f = ((z0[k] + 0.5 * dz_[k]) * x0[i] + (0.5 * z0[k] + third * dz_[k]) * dx_[i])
                J[1].index_add_(0, ix[i] * n[2] + iz[k], f * (-w * vy / (d[0] * d[2])))
            for i, cu in enumerate(cum(dx_)):
                J[0].index_add_(0, ix[i] * n[2] + iz[k], cx * cu * (z0[k] + 0.5 * dz_[k]))
        for i in range(M):
            for k, cu in enumerate(cum(dz_)):
                J[2].index_add_(0, ix[i] * n[2] + iz[k], cz * cu * (x0[i] + 0.5 * dx_[i]))
        return [a.view(n) for a in J]
    by, y0, y1 = _box(order, new[1], old[1])
    iy = _axis(n[1], by, M)
    dy_ = [b - a for a, b in zip(y0, y1)]
    S0, D, I = (x0, y0, z0), (dx_, dy_, dz_), (ix, iy, iz)
    area = (dt * d[1] * d[2], dt * d[0] * d[2], dt * d[0] * d[1])
    flat = lambda i, j, k: (i * n[1] + j) * n[2] + k
    for a in range(3):
        p, q = [t for t in range(3) if t != a]
        C = [v * (-w / area[a]) for v in cum(D[a])]
        for r in range(M):
            for t in range(M):
                f = ((S0[p][r] + 0.5 * D[p][r]) * S0[q][t] +
                     (0.5 * S0[p][r] + D[p][r] / 3.0) * D[q][t])
                for e in range(M - 1):
                    at = [None] * 3
                    at[a], at[p], at[q] = I[a][e], I[p][r], I[q][t]
                    J[a].index_add_(0, flat(*at), C[e] * f)
    return [a.view(n) for a in J]


_FD = {2: (1.0,), 4: (9.0 / 8.0, -1.0 / 24.0)}


def _diff(f, a, norder, forward):
    """Staggered difference along axis a: forward f[i+1] - f[i] or backward."""
    if f.shape[a] == 1:
        return torch.zeros_like(f)
    out = torch.zeros_like(f)
    for l, w in enumerate(_FD[norder], 1):
        hi, lo = (-l, l - 1) if forward else (-(l - 1), l)
        out += w * (torch.roll(f, hi, a) - torch.roll(f, lo, a))
    return out


def _curl(F, d, norder, forward):
    D = lambda f, a: _diff(f, a, norder, forward) / d[a]
    return [D(F[2], 1) - D(F[1], 2), D(F[0], 2) - D(F[2], 0), D(F[1], 0) - D(F[0], 1)]


def _pic(E, B, pos, u, w, d, dt, order, pusher, steps, norder=2):
    """steps periodic PIC steps; positions in cells.  Returns E, B, J, pos, u."""
    n = tuple(E[0].shape)
    J = None
    for _ in range(steps):
        eb = _gather(E + B, pos, order, True)
        u, gi = (_vay if pusher == 1 else _boris)(u, eb, dt)
        move = [a * gi * dt / h for a, h in zip(u, d)]
        if n[1] == 1:
            move[1] = torch.zeros_like(w)
        new = [a + b for a, b in zip(pos, move)]
        J = _deposit(n, new, pos, w, d, dt, order, u[1] * gi)
        pos = [torch.where(a < 0, a + v, torch.where(a >= v, a - v, a)) for a, v in zip(new, n)]
        B = [b - 0.5 * dt * c for b, c in zip(B, _curl(E, d, norder, True))]
        E = [e + dt * (c - j) for e, c, j in zip(E, _curl(B, d, norder, False), J)]
        B = [b - 0.5 * dt * c for b, c in zip(B, _curl(E, d, norder, True))]
    return E, B, J, pos, u


def _cfl(d, dims=3, coef=0.95):
    return coef / math.sqrt(sum(1.0 / v ** 2 for v in (d if dims == 3 else (d[0], d[2]))))


def _exact_jobs(specs, steps):
    """The outputs of an ensemble's jobs of one shape order.

    FP32 at order 1 has no such value: the staggered order-1 shape is a step
    of the position, so a particle within rounding of a cell edge takes
    another cell's field, and the distance from 64 bits counts such particles
    and not the digits of the rest."""
    outs = []
    for sp in specs:
        st = thermal_plasma(sp.n, sp.ppc, sp.sigma, seed=sp.seed, device="cuda")
        z = [torch.zeros(sp.n, dtype=torch.float64, device="cuda") for _ in range(6)]
        outs.append(_pic(z[:3], z[3:], [st.x, st.y, st.z], [st.ux, st.uy, st.uz], st.w,
                         (1.0, 1.0, 1.0), _cfl((1.0, 1.0, 1.0)), sp.order, sp.pusher, steps))
    r = {name: torch.cat([_guarded((E + B)[q]).permute(2, 1, 0).reshape(-1)
                          for E, B, _, _, _ in outs]) for q, name in enumerate(EB)}
    r.update((name, torch.cat([(pos + u)[q] for _, _, _, pos, u in outs]))
             for q, name in enumerate(COLS))
    r.update((k, _moved(r[k], *b)) for k, b in zip(COLS[:3], _starts(specs)))
    return r


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "ensemble":
        return {"order%d" % o: _exact_jobs(v, c["steps"]) if o > 1 else None
                for o, v in _by_order(_specs(c, seed), lambda t: t.order).items()}
    if kind == "tiled" and c["precision"] == "fp32" and c["order"] == 1:
        return None                                       # see _exact_jobs
    np_ = _particles(c)
    if np_ * c.get("steps", 1) * c["order"] ** 3 > 1.2e10:     # over about 20 s
        return None
    st, n, d = _plasma(c, seed), _n(c), _d(c)
    F = _waves(n, seed, c["order"])
    if kind == "module2d":
        st.y.zero_()
    pos, u = [st.x / d[0], st.y / d[1], st.z / d[2]], [st.ux, st.uy, st.uz]
    if kind == "routines":
        gi = 1.0 / torch.sqrt(1.0 + sum(a ** 2 for a in u))
        eb = _gather(F, pos, c["order"], c["lower"])
        # the routine deposits the move that ended at pos, unfolded at the
        # edges: the outer guard nodes hold what falls there
        g = 4
        wide = tuple(v + 2 * g + 1 for v in n)
        new = [a + g for a in pos]
        old = [a - 0.5 * b * gi for a, b in zip(new, u)]
        J = _deposit(wide, new, old, st.w, d, 0.5, c["order"])
        return dict(zip(EB + J3, eb + J))
    coef = 0.8 if c.get("norder", 2) > 2 else 0.95
    dt = _cfl(d, 2 if kind == "module2d" else 3, coef)
    E, B, J, pos, u = _pic(F[:3], F[3:], pos, u, st.w, d, dt, c["order"], c["pusher"], c["steps"],
                           c.get("norder", 2))
    out = {name: _guarded(f) for name, f in zip(EB + J3, E + B + J)}
    out.update(zip(COLS, [a * h for a, h in zip(pos, d)] + u))
    if kind == "tiled":
        for name in J3:
            del out[name]
        out.update((k, _moved(out[k], a, float(v)))
                   for k, a, v in zip(COLS, (st.x, st.y, st.z), n))
    return out
