"""The workloads whose speed this framework is judged by, through its public Python face.

A case is one pass of a user's program:

* ``step``    one building: n gas-phase steps (Solver.run) and the state read back,
              as a case run does between two outputs;
* ``batch``   several buildings stepped together (Batch.step), each with its own
              dtMax, and their states read back, as a what-if or training-data
              service does between two samplings;
* ``rad``     one radiation trace over the resident gas fields (Solver.rad_trace),
              as a coupled run does every radiation interval;
* ``render``  one frame of the smoke and flame volume (Solver.vol_render), as the
              viewer or a film of a run does.

The states are developed fires made from the seed (a hot plume over the burner, a
layer under the ceiling, a smooth eddying flow); the buildings are those of
photon_gb300.casegen. The pressure solve stops at a relative residual of 1e-8.
Fields of a mixed context are returned in FP32, the type the context keeps them in.

`exact` restates the step and the trace in torch in FP64, with a Jacobi-preconditioned
CG that runs to a relative residual of 1e-12. A frame has no 64-bit value: its dither
is the fractional part of a large FP32 product.
"""
import math

import numpy as np
import torch

from photon_gb300 import _lib, casegen, render
from photon_gb300.solver import Batch, Solver

STATE = ("u", "v", "w", "p", "T", "Yo", "Yf", "Ys", "Ya", "Yp", "Yc", "Yw", "Yco", "Yai")
REL_TOL = 1e-8
DT_MAX = 0.02
T0 = 293.15


def listed():
    return [
        # the smallest call: one step of a 1,287-cell closet with a doorway, read back at once
        # (an interactive session, a unit test); odd sizes
        {"name": "closet-step-fp64", "kind": "step", "room": "tiny", "nx": 13, "ny": 11, "nz": 9, "dx": 0.2,
         "precision": "fp64", "steps": 1, "wind": 0.0, "house": 0},
        # the single room of the reference's tests, 36x24x24, in both precisions
        {"name": "room-run-fp64", "kind": "step", "room": "single", "nx": 36, "ny": 24, "nz": 24, "dx": 0.1,
         "precision": "fp64", "steps": 20, "wind": 0.0, "house": 0},
        {"name": "room-run-mixed", "kind": "step", "room": "single", "nx": 36, "ny": 24, "nz": 24, "dx": 0.1,
         "precision": "mixed", "steps": 20, "wind": 0.0, "house": 0},
        # the 72x52x44 house at 0.2 m, in both precisions
        {"name": "house-run-fp64", "kind": "step", "room": "house", "nx": 72, "ny": 52, "nz": 44, "dx": 0.2,
         "precision": "fp64", "steps": 20, "wind": 0.0, "house": 1},
        {"name": "house-run-mixed", "kind": "step", "room": "house", "nx": 72, "ny": 52, "nz": 44, "dx": 0.2,
         "precision": "mixed", "steps": 20, "wind": 0.0, "house": 1},
        # a house with odd sizes in a wind (inflow faces closed in the pressure matrix)
        {"name": "windy-house-mixed", "kind": "step", "room": "house", "nx": 61, "ny": 47, "nz": 31, "dx": 0.2,
         "precision": "mixed", "steps": 20, "wind": 4.0, "house": 7},
        # the largest single building: the same house at 0.1 m, 1.32 M cells
        {"name": "fine-house-run-mixed", "kind": "step", "room": "house", "nx": 144, "ny": 104, "nz": 88, "dx": 0.1,
         "precision": "mixed", "steps": 20, "wind": 0.0, "house": 1},
        # batches of seeded houses of 20 k to 400 k cells, as the throughput benchmark draws them
        {"name": "batch24-mixed", "kind": "batch", "scenarios": 24, "lo": 20000, "hi": 400000, "house": 2024,
         "precision": "mixed", "steps": 40},
        {"name": "batch8-fp64", "kind": "batch", "scenarios": 8, "lo": 20000, "hi": 160000, "house": 2024,
         "precision": "fp64", "steps": 20},
        # radiation traces: the fine house in the mixed path's FP32, the coarse one in FP64
        {"name": "fine-house-trace-mixed", "kind": "rad", "nx": 144, "ny": 104, "nz": 88, "dx": 0.1,
         "precision": "mixed", "house": 1},
        {"name": "house-trace-fp64", "kind": "rad", "nx": 72, "ny": 52, "nz": 44, "dx": 0.2,
         "precision": "fp64", "house": 1},
        # a 1280x720 frame of the house: smoke, fire and a temperature slice
        {"name": "house-frame-720p", "kind": "render", "nx": 72, "ny": 52, "nz": 44, "dx": 0.2, "house": 1,
         "width": 1280, "height": 720, "slice": True, "precision": "mixed"},
    ]


def _dims(rng, cells):
    """Sides of a grid of about `cells` cells, aspect ratios of 1-3, the height the smallest; at least 12."""
    ar = math.exp(rng.uniform(0.0, math.log(3.0)))
    a2 = math.exp(rng.uniform(0.0, math.log(ar)))
    base = (cells / (ar * a2)) ** (1.0 / 3.0)
    nx, ny, nz = round(base * ar), round(base * a2), round(base)
    return max(nx, 12), max(ny, 12), max(nz, 9)


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    pick = rng.random()
    precision = "mixed" if rng.random() < 0.6 else "fp64"
    house = rng.randrange(1 << 20)
    dx = rng.choice((0.1, 0.2))
    if pick < 0.6:
        cells = _log(rng, 1.5e3, 1.2e6 if precision == "mixed" else 1.6e5)
        nx, ny, nz = _dims(rng, cells)
        big = nx >= 20 and ny >= 20 and nz >= 16
        room = "house" if big and rng.random() < 0.75 else "tiny"
        # a wind needs a way out: the closet's only opening would be its inflow
        wind = rng.uniform(1.0, 8.0) if room == "house" and rng.random() < 0.33 else 0.0
        return {"kind": "step", "room": room, "nx": nx, "ny": ny, "nz": nz, "dx": dx, "precision": precision,
                "steps": rng.randint(1, 20), "wind": wind, "house": house}
    if pick < 0.75:
        mixed = precision == "mixed"
        return {"kind": "batch", "scenarios": rng.randint(2, 24 if mixed else 8), "lo": 20000,
                "hi": round(_log(rng, 4e4, 4e5 if mixed else 1.6e5)), "house": house, "precision": precision,
                "steps": rng.randint(5, 40 if mixed else 20)}
    if pick < 0.9:
        nx, ny, nz = _dims(rng, _log(rng, 1e4, 1.2e6 if precision == "mixed" else 1.6e5))
        return {"kind": "rad", "nx": max(nx, 20), "ny": max(ny, 20), "nz": max(nz, 16), "dx": dx,
                "precision": precision, "house": house}
    nx, ny, nz = _dims(rng, _log(rng, 1e4, 1.6e5))
    h = rng.randint(180, 720)
    return {"kind": "render", "nx": max(nx, 20), "ny": max(ny, 20), "nz": max(nz, 16), "dx": dx, "house": house,
            "width": round(h * rng.uniform(1.2, 1.78)), "height": h, "slice": rng.random() < 0.5,
            "precision": precision}


# ---- buildings and states ------------------------------------------------------------

def _profile():
    p = casegen.Profile.reference()
    p.tol, p.rel_tol = 1e-12, REL_TOL     # the relative stop decides
    return p


def _building(case):
    """The casegen.Case of a one-building case."""
    room = case.get("room", "house")
    if room == "single":
        c = casegen.single_room(profile=_profile())
    elif room == "tiny":
        c = casegen.tiny_room(case["nx"], case["ny"], case["nz"], case["dx"])
        c.profile = _profile()
    else:
        c = casegen.house(case["nx"], case["ny"], case["nz"], case["dx"], case["house"], profile=_profile())
    if case.get("wind", 0.0) > 0:
        c.wind = (case["wind"], 250.0, 0.25)
    return c


def _buildings(case):
    if case["kind"] != "batch":
        return [_building(case)]
    cs = casegen.batch_scenarios(case["scenarios"], case["house"], case["lo"], case["hi"])
    for c in cs:
        c.profile = _profile()
    return cs


def _waves(rng, xyz, amplitude, lengths):
    """A smooth random field: a few plane waves of the given lengths (m)."""
    out = 0.0
    for length in lengths:
        k = rng.normal(size=3)
        k *= 2.0 * np.pi / length / np.linalg.norm(k)
        x = [np.exp(1j * k[a] * xyz[a]) for a in range(3)]
        plane = (x[1][:, None] * x[0][None, :])[None] * (x[2] * np.exp(2j * np.pi * rng.random()))[:, None, None]
        out = out + amplitude * plane.real
    return out


def _fire_state(c, seed):
    """A developed fire in building c: the fields of STATE by name, and the elapsed time."""
    rng = np.random.default_rng([seed, c.nx, c.ny, c.nz])
    nx, ny, nz, dx = c.nx, c.ny, c.nz, c.dx
    b = c.blocked.reshape(nz, ny, nx) != 0
    xc = [o + (np.arange(n) + 0.5) * dx for o, n in ((c.ox, nx), (c.oy, ny), (c.oz, nz))]
    xf = [o + np.arange(n + 1) * dx for o, n in ((c.ox, nx), (c.oy, ny), (c.oz, nz))]
    bu = c.burners[0]
    px, py = 0.5 * (bu.x0 + bu.x1), 0.5 * (bu.y0 + bu.y1)
    r2 = (xc[0][None, :] - px) ** 2 + (xc[1][:, None] - py) ** 2
    z = (xc[2] - c.oz)[:, None, None]
    width = 0.3 + 0.12 * z
    plume = np.exp(-r2[None] / width**2) * np.clip(1.1 - 0.25 * z, 0.1, 1.0)
    ceiling = min(2.4, nz * dx)
    layer = np.clip((z - 0.5 * ceiling) / (0.5 * ceiling), 0.0, 1.0) * 0.3 * np.exp(-r2[None] / 30.0)
    layer = np.where(z < ceiling, layer, 0.0)
    heat = np.clip(np.maximum(plume, layer) * (1.0 + _waves(rng, xc, 0.05, (0.9, 1.7, 3.1))), 0.0, 1.2)
    fuel = 0.03 * np.clip(plume - 0.3, 0.0, 1.0) ** 2
    gas = {"T": T0 + 850.0 * heat, "Yo": 0.232 * (1.0 - 0.6 * np.minimum(heat, 1.0)), "Yf": fuel, "Ys": 0.003 * heat,
           "Ya": 0.0005 * heat, "Yp": 0.01 * fuel, "Yc": 0.0006 + 0.07 * heat, "Yw": 0.0073 + 0.05 * heat,
           "Yco": 0.002 * heat, "Yai": 800.0 * fuel}
    amb = {"T": T0, "Yo": 0.232, "Yc": 0.0006, "Yw": 0.0073}
    state = {k: np.where(b, amb.get(k, 0.0), v) for k, v in gas.items()}
    state["p"] = np.where(b, 0.0, _waves(rng, xc, 0.1, (2.0, 4.0)))
    for a, (name, f) in enumerate((("u", c.fx), ("v", c.fy), ("w", c.fz))):
        xyz = list(xc)
        xyz[a] = xf[a]
        shape = [nz, ny, nx]
        shape[2 - a] += 1
        vel = _waves(rng, xyz, 0.25, (0.7, 1.5, 3.0, 6.0))
        if a == 2:
            up = np.concatenate([plume[:1], 0.5 * (plume[1:] + plume[:-1]), plume[-1:]])
            vel = vel + 2.5 * up
        state[name] = np.where(f.reshape(shape) > 0, vel, 0.0)
    return {k: np.ascontiguousarray(v.reshape(-1)) for k, v in state.items()}, 30.0 + 10.0 * rng.random()


def _load(put, set_stats, state, time):
    for f in STATE:
        put(f, state[f])
    speed = max(float(np.abs(state[f]).max()) for f in "uvw")
    set_stats({"time": time, "max_vel": speed, "max_nu": 0.0, "max_div": 0.0, "hrr": 0.0, "max_gas_t": T0,
               "burning_cells": 0, "fuel_in": 0.0, "fuel_burned": 0.0, "fuel_in_domain": 0.0})
    return speed


def _set_batch_stats(b, s, st):
    rec = _lib.PhxStats()
    for k, v in st.items():
        setattr(rec, k, v)
    b._check(b.L.phx_batch_set_stats(b.h, s, rec))


def _trace_inputs(c, case, seed):
    """The trace's inputs: the surfaces are the building's, their temperatures and the gas the seed's."""
    w = casegen.rad_workload(c, case["house"])
    rng = np.random.default_rng(seed)
    gas = dict(w["gas"])
    b = c.blocked != 0
    scale = 1.0 + 0.1 * (rng.random(c.N) - 0.5)
    gas["T"] = np.where(b, T0, T0 + (gas["T"] - T0) * scale)
    for k in ("Ys", "Yc", "Yw"):
        gas[k] = gas[k] * scale
    el, wl = w["elements"].copy(), w["walls"].copy()
    el[:, 8] = T0 + (el[:, 8] - T0) * rng.uniform(0.8, 1.2, len(el))
    wl[:, 2:4] = T0 + (wl[:, 2:4] - T0) * rng.uniform(0.8, 1.2, (len(wl), 2))
    solid = T0 + (w["solidT"] - T0) * rng.uniform(0.8, 1.2, c.N)
    return {"gas": gas, "elements": el, "walls": wl, "solidT": solid}


def _precision(case):
    return _lib.PREC_MIXED if case["precision"] == "mixed" else _lib.PREC_FP64


def _step_limits(n):
    """The dtMax of each building of a batch (each run has its own output times)."""
    return np.array([DT_MAX * (1.0 - 0.02 * (s % 8)) for s in range(n)])


def prepare(case, seed):
    out = {"kind": case["kind"], "real": np.float32 if case["precision"] == "mixed" else np.float64}
    cs = _buildings(case)
    if case["kind"] == "batch":
        b = Batch(cs, _precision(case))
        for s, c in enumerate(cs):
            state, time = _fire_state(c, seed)
            _load(lambda f, a, s=s: b.set(s, f, a), lambda st, s=s: _set_batch_stats(b, s, st), state, time)
        return out | {"batch": b, "steps": case["steps"], "limits": _step_limits(len(cs))}
    c = cs[0]
    s = Solver(c, _precision(case))
    out["solver"] = s
    state, time = _fire_state(c, seed)
    if case["kind"] == "rad":
        w = _trace_inputs(c, case, seed)
        for k, v in w["gas"].items():
            s.set(k, v)
        out |= {k: w[k] for k in ("elements", "walls", "solidT")}
    else:
        _load(s.set, s.set_stats, state, time)
    if case["kind"] == "step":
        out["steps"] = case["steps"]
    elif case["kind"] == "render":
        rng = np.random.default_rng(seed)
        hrr = 2.0e6 * np.clip(state["T"] - 800.0, 0.0, 400.0) / 400.0
        s.set("hrr", hrr)
        size = np.array([c.nx, c.ny, c.nz]) * c.dx
        eye = np.array([c.ox, c.oy, c.oz]) + size * np.array([-0.3, -0.4, 0.8]) + 0.2 * rng.random(3)
        target = np.array([c.ox, c.oy, c.oz]) + size * np.array([0.5, 0.5, 0.25])
        out["camera"] = render.camera(c, eye, target, case["width"], case["height"], time=time,
                                      slice_z=c.oz + 1.2 if case["slice"] else None,
                                      lights=render.fire_lights(c, hrr, time))
    return out


def run(state):
    kind, real = state["kind"], state["real"]
    if kind == "step":
        s = state["solver"]
        dt = s.run(state["steps"], DT_MAX)
        return {"dt": dt.astype(real)} | {f: s.get(f).astype(real, copy=False) for f in STATE}
    if kind == "batch":
        b = state["batch"]
        dt = np.stack([b.step(state["limits"]) for _ in range(state["steps"])])
        out = {"dt": dt.astype(real)}
        for f in STATE:
            out[f] = np.concatenate([b.get(s, f).astype(real, copy=False) for s in range(len(b))])
        return out
    s = state["solver"]
    if kind == "rad":
        absorbed, gas = s.rad_trace(state["elements"], state["walls"], state["solidT"])
        return {"absorbed": absorbed.astype(real), "gas": gas.astype(real)}
    return {"rgb": s.vol_render(state["camera"])}


def work(case):
    """Per step, a cell's 14 state values are read and written, its three open fractions and its solid flag read,
    and about 3,000 operations done (ten limited scalars, momentum, a solve of a few multigrid cycles); a trace reads
    its elements, walls and gas once; a frame reads the volume and writes its pixels."""
    w = 4 if case["precision"] == "mixed" else 8
    if case["kind"] in ("step", "batch"):
        if case["kind"] == "step":
            n = case["nx"] * case["ny"] * case["nz"]
        else:   # log-uniform sizes
            n = case["scenarios"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": n * case["steps"] * (31.0 * w + 1.0), "flops": n * case["steps"] * 3000.0}
    n = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "rad":
        # about 0.16 elements and 0.06 walls per cell, 17 rays per element, some 8 cells per ray, 60 operations each
        return {"bytes": n * (7.0 * w + 8.0 + 0.16 * 96.0 + 0.06 * 24.0), "flops": n * 0.16 * 17 * 8 * 60.0}
    # a ray samples a few dozen points, each a trilinear read of four values
    return {"bytes": n * 16.0 + case["width"] * case["height"] * 12.0,
            "flops": case["width"] * case["height"] * 40 * 100.0}


# ---- the same in 64 bits -------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _shift(a, axis, by, fill):
    """a moved so that element i holds a[i + by] along `axis`; `fill` (a number or a tensor like a) past the end."""
    n = a.shape[axis]
    out = fill.clone() if torch.is_tensor(fill) else torch.full_like(a, fill)
    m = n - abs(by)
    if m > 0:
        out.narrow(axis, max(0, -by), m).copy_(a.narrow(axis, max(0, by), m))
    return out


def _inside(a, axis):
    return a.narrow(axis, 1, a.shape[axis] - 2)


def _superbee_times(num, den, floor):
    """superbee(num / den) den, 0 where |den| is at most `floor`."""
    safe = torch.where(den.abs() > floor, den, torch.ones_like(den))
    r = num / safe
    lim = torch.maximum(torch.clamp(torch.minimum(2 * r, torch.ones_like(r)), min=0.0),
                        torch.minimum(r, torch.full_like(r, 2.0)))
    return torch.where(den.abs() > floor, lim * den, torch.zeros_like(den))


class _Room64:
    """The gas-phase step of one building whose zones are all open to the atmosphere, in FP64: arrays are
    [nz, ny, nx]; axis a of the grid (x, y, z) is dimension 2 - a."""

    P0, RS, CP, G = 101325.0, 287.0, 1100.0, 9.81
    AMB = {"T": T0, "Yo": 0.232, "Yc": 0.0006, "Yw": 0.0073}
    SCALARS = ("T", "Yo", "Yf", "Ys", "Ya", "Yp", "Yc", "Yw", "Yco", "Yai")

    def __init__(self, c, state, time, speed):
        self.c, self.dx, self.time = c, c.dx, time
        dev = _device()
        put = lambda a, shape: torch.tensor(np.asarray(a, np.float64).reshape(shape), device=dev)
        self.n = n = (c.nx, c.ny, c.nz)
        self.shape = (c.nz, c.ny, c.nx)
        fshape = [[c.nz, c.ny, c.nx + 1], [c.nz, c.ny + 1, c.nx], [c.nz + 1, c.ny, c.nx]]
        self.f = {k: put(state[k], self.shape) for k in self.SCALARS + ("p",)}
        self.vel = [put(state[k], fshape[a]) for a, k in enumerate("uvw")]
        self.open = [put(x, fshape[a]) for a, x in enumerate((c.fx, c.fy, c.fz))]
        self.blocked = put(c.blocked, self.shape) > 0
        self.lit = torch.zeros_like(self.blocked)
        self.max_vel, self.max_nu, self.max_div = speed, 0.0, 0.0
        zc = c.oz + (torch.arange(c.nz, dtype=torch.float64, device=dev) + 0.5) * c.dx
        self.wind = [[self._wind(a, side, zc) for side in (0, 1)] for a in range(2)]
        # matrix coefficients: the open fractions with wind-inflow faces closed
        self.a0 = [x.clone() for x in (put(c.ax, fshape[0]), put(c.ay, fshape[1]), put(c.az, fshape[2]))]
        for a in range(2):
            for side in (0, 1):
                if self.wind[a][side] is not None:
                    self.a0[a].select(2 - a, n[a] if side else 0).zero_()
        self.am = [put(x, fshape[a]) for a, x in enumerate((c.ax, c.ay, c.az))]
        self.diag = sum(self._lo(a, self.a0[a]) + self._hi(a, self.a0[a]) for a in range(3))
        self.diag = torch.where(self.blocked, torch.zeros_like(self.diag), self.diag)
        self.burners = [self._burner(b) for b in c.burners]

    # face arrays seen from the cells below / above them
    def _lo(self, a, f):
        return f.narrow(2 - a, 0, self.n[a])

    def _hi(self, a, f):
        return f.narrow(2 - a, 1, self.n[a])

    def _wind(self, axis, side, zc):
        """Inflow speed of a domain side, per layer, or None where the side is open."""
        speed, deg, ex = self.c.wind
        if speed <= 0:
            return None
        th = deg * 3.14159265 / 180.0
        comp = (-math.sin(th) if axis == 0 else -math.cos(th)) * speed * (torch.clamp(zc, min=0.05) / 10.0) ** ex
        if (float(comp[0]) > 0) == (side == 0) and float(comp[0]) != 0:
            return comp[:, None]
        return None

    def _burner(self, b):
        c = self.c
        x = c.ox + (np.arange(c.nx) + 0.5) * c.dx
        y = c.oy + (np.arange(c.ny) + 0.5) * c.dx
        m = np.zeros(self.shape, bool)
        k = int(math.floor((b.z + 0.5 * c.dx - c.oz) / c.dx))
        m[k] = ((y >= b.y0) & (y <= b.y1))[:, None] & ((x >= b.x0) & (x <= b.x1))[None]
        m &= c.blocked.reshape(self.shape) == 0
        if not m.any():
            i, j = (int(math.floor((0.5 * s - o) / c.dx)) for s, o in ((b.x0 + b.x1, c.ox), (b.y0 + b.y1, c.oy)))
            m[k, j, i] = True
        return torch.tensor(m, device=self.diag.device), int(m.sum())

    def open_zones_only(self):
        """Whether every gas cell is connected to an open face of the domain."""
        reach = torch.zeros_like(self.blocked)
        for a in range(3):
            ends = [(0, self._lo), (self.n[a] - 1, self._hi)]
            for at, side in ends[1:] if a == 2 else ends:
                sel = side(a, self.am[a]).select(2 - a, at) > 0
                reach.select(2 - a, at).logical_or_(sel)
        reach &= ~self.blocked
        while True:
            grown = reach.clone()
            for a in range(3):
                for by, side in ((1, self._hi), (-1, self._lo)):
                    grown |= _shift(reach, 2 - a, by, False) & (side(a, self.am[a]) > 0)
            grown &= ~self.blocked
            if bool((grown == reach).all()):
                return bool((reach | self.blocked).all())
            reach = grown

    def rho(self):
        return self.P0 / (self.RS * self.f["T"])

    def stable_dt(self, limit):
        dt = min(limit, self.c.profile.dtMax, self.c.profile.cfl * self.dx / max(self.max_vel, 0.1))
        alpha = self.max_nu * (1.0 + 1.0 / 0.5)
        if alpha > 0:
            dt = min(dt, 0.9 * self.dx * self.dx / (6.0 * alpha))
        if self.max_div > 0:
            dt = min(dt, 0.25 / self.max_div)
        return max(dt, 1e-3)

    def combust(self, dt):
        f, dx = self.f, self.dx
        zero = torch.zeros_like(f["T"])
        self.Q, self.mass = zero.clone(), zero.clone()
        pilot = torch.zeros_like(self.blocked)
        for (m, cells), b in zip(self.burners, self.c.burners):
            on = b.start <= self.time <= b.start + b.duration
            ramp = min(1.0, (self.time - b.start) / b.rampS) if b.rampS > 0 else 1.0
            mf = b.peakW * ramp * ramp * dt / 25.0e6 / cells if on else 0.0
            if mf <= 0:
                continue
            mass = self.rho() * dx**3
            mt = mass + mf
            scl = mass / mt
            for k, gain in (("Yo", 0.0), ("Ys", 0.0), ("Yc", 0.0), ("Yw", 0.0), ("Yco", 0.0), ("Yai", 800.0 * mf),
                            ("Yf", mf), ("Ya", 0.0), ("Yp", 0.01 * mf)):
                f[k] = torch.where(m, f[k] * scl + gain / mt, f[k])
            self.mass = self.mass + m * mf
            pilot |= m
        frac = 1.0 - math.exp(-dt / 0.1)
        chi = 0.35 if self.c.radiationOn else 0.0
        yf, yo, Tc = f["Yf"], f["Yo"], f["T"]
        ait = torch.where(yf > 1e-9, f["Yai"] / torch.clamp(yf, min=1e-30), torch.full_like(yf, 800.0))
        near = torch.zeros_like(self.lit)
        for a in range(3):
            for by in (1, -1):
                near |= _shift(self.lit, 2 - a, by, False)
        burnable = torch.minimum(yf, yo / 1.95)
        t_ad = Tc + 25.0e6 / (1100.0 * (1.0 + 1.95 / torch.clamp(yo, min=1e-4)))
        go = ~self.blocked & (yf >= 1e-6) & (pilot | (Tc > ait) | near) & (burnable > 1e-7) & (pilot | ~(t_ad < 1600.0))
        m = self.rho() * dx**3
        dmf = burnable * m * frac
        q = dmf * 25.0e6
        soot = torch.where(yf > 0, f["Yp"] * (dmf / m) / torch.clamp(yf, min=1e-30), zero)
        co = 0.02 * dmf / m
        co2 = torch.clamp((0.597 * dmf / m - soot - (12.0 / 28.0) * co) * (44.0 / 12.0), min=0.0)
        o2 = 1.95 * dmf / m - (32.0 / 12.0) * soot - (16.0 / 28.0) * co
        new = {"Yf": torch.clamp(yf - dmf / m, min=0.0), "Yo": torch.clamp(yo - o2, min=0.0),
               "Yp": torch.clamp(f["Yp"] - soot, min=0.0), "Ys": f["Ys"] + soot, "Yco": f["Yco"] + co,
               "Yc": f["Yc"] + co2, "Yw": f["Yw"] + 0.761 * dmf / m, "Ya": f["Ya"] * (1.0 - frac)}
        new["Yai"] = new["Yf"] * ait
        for k, v in new.items():
            f[k] = torch.where(go, v, f[k])
        self.Q = torch.where(go, q * (1.0 - chi), self.Q)
        self.lit = go & (q > 1e-3)

    def turbulence(self):
        gas = ~self.blocked
        ks = 0.0
        for a in range(3):
            v = torch.where(gas, 0.5 * (self._lo(a, self.vel[a]) + self._hi(a, self.vel[a])), torch.zeros_like(self.diag))
            s = v
            for d in range(3):
                lo = torch.where(_shift(gas, 2 - d, -1, False), _shift(s, 2 - d, -1, 0.0), s)
                hi = torch.where(_shift(gas, 2 - d, 1, False), _shift(s, 2 - d, 1, 0.0), s)
                s = torch.where(gas, 0.25 * lo + 0.5 * s + 0.25 * hi, torch.zeros_like(s))
            ks = ks + (v - s) ** 2
        nu = 0.1 * self.dx * torch.sqrt(0.5 * ks) + 1.5e-5 * (self.f["T"] / 293.15) ** 1.7
        self.nu = torch.where(gas, torch.clamp(nu, max=1.0), torch.zeros_like(nu))
        self.max_nu = float(self.nu.max())

    def neighbours(self):
        """Per face of a cell (x-, x+, ...): axis, shift, its open fraction, whether the neighbour is in the domain,
        and whether heat and matter pass (open, no solid behind)."""
        for a in range(3):
            for by, side in ((-1, self._lo), (1, self._hi)):
                fo = side(a, self.open[a])
                inside = _shift(torch.ones_like(self.blocked), 2 - a, by, False)
                yield a, by, fo, inside, (fo > 0) & ~_shift(self.blocked, 2 - a, by, False)

    def heat_and_energy(self, dt):
        T, rho, dx = self.f["T"], self.rho(), self.dx
        q = torch.zeros_like(T)
        for a, by, fo, inside, on in self.neighbours():
            Tn = _shift(T, 2 - a, by, T0)
            nun = torch.where(inside, _shift(self.nu, 2 - a, by, 0.0), self.nu)
            rn = _shift(rho, 2 - a, by, self.P0 / (self.RS * T0))
            kf = 0.5 * (rho + rn) * self.CP * 0.5 * (self.nu + nun) / 0.5 + 0.0258 * (0.5 * (T + Tn) / 293.15) ** 0.8
            q = q + torch.where(on, fo * kf * dx * (Tn - T), torch.zeros_like(q))
        gas, V = ~self.blocked, dx**3
        Q = self.Q + q * dt
        m = rho * V
        Tn = torch.clamp(T + Q / (m * self.CP), 200.0, 2300.0)
        D = Q / (m * self.CP * T * dt) + self.mass / (self.P0 / (self.RS * Tn) * V * dt)
        self.S = torch.where(gas, torch.clamp(D, -50.0, 50.0), torch.zeros_like(D))
        self.max_div = float(self.S.abs().max())
        self.f["T"] = torch.where(gas, Tn, T)

    def momentum(self, dt):
        rho, dx, new = self.rho(), self.dx, []
        centre = [0.5 * (self._lo(a, self.vel[a]) + self._hi(a, self.vel[a])) for a in range(3)]
        for a in range(3):
            dim, v0, fo = 2 - a, self.vel[a], self.open[a]
            n = self.n[a]
            pair = lambda x: (x.narrow(dim, 0, n - 1), x.narrow(dim, 1, n - 1))   # the cells beside an interior face
            acc, lap = 0.0, 0.0
            vi = _inside(v0, dim)
            for d in range(3):
                adv = vi if d == a else 0.5 * sum(pair(centre[d]))
                ok = fo > 0
                m1o, p1o = _shift(ok, 2 - d, -1, False), _shift(ok, 2 - d, 1, False)
                m2o, p2o = _shift(ok, 2 - d, -2, False) & m1o, _shift(ok, 2 - d, 2, False) & p1o
                m1 = torch.where(m1o, _shift(v0, 2 - d, -1, 0.0), v0)
                p1 = torch.where(p1o, _shift(v0, 2 - d, 1, 0.0), v0)
                m2 = torch.where(m2o, _shift(v0, 2 - d, -2, 0.0), m1)
                p2 = torch.where(p2o, _shift(v0, 2 - d, 2, 0.0), p1)
                m1, p1, m2, p2 = (_inside(x, dim) for x in (m1, p1, m2, p2))

                def van_leer(x, y):
                    pos = x * y > 0
                    return torch.where(pos, 2 * x * y / torch.where(pos, x + y, torch.ones_like(x)), torch.zeros_like(x))

                fp = torch.where(adv >= 0, vi + 0.5 * van_leer(vi - m1, p1 - vi), p1 - 0.5 * van_leer(p1 - vi, p2 - p1))
                fm = torch.where(adv >= 0, m1 + 0.5 * van_leer(m1 - m2, vi - m1), vi - 0.5 * van_leer(vi - m1, p1 - vi))
                acc = acc - adv * (fp - fm) / dx
                lap = lap + (m1 - 2 * vi + p1) / (dx * dx)
            ra, rb = pair(rho)
            rf = 0.5 * (ra + rb)
            acc = acc + 0.5 * sum(pair(self.nu)) * lap
            if a == 2:
                acc = acc + self.G * (self.P0 / (self.RS * T0) - rf) / rf
            acc = acc + rf * 0.5 * sum(pair(self.f["p"])) * (1.0 / rb - 1.0 / ra) / dx
            out = v0.clone()
            _inside(out, dim).copy_(torch.clamp(vi + dt * acc, -40.0, 40.0))
            out = torch.where(fo > 0, out, torch.zeros_like(out))
            for side, at, inner in ((0, 0, 1), (1, n, n - 1)):
                if a == 2 and side == 0:
                    continue
                w = self.wind[a][side] if a < 2 else None
                value = out.select(dim, inner).clone() if w is None else w.expand_as(out.select(dim, at))
                face = out.select(dim, at)
                face.copy_(torch.where(fo.select(dim, at) > 0, value, torch.zeros_like(value)))
            new.append(out)
        self.vel = new

    def _apply(self, x):
        s = self.diag * x
        for a in range(3):
            inner = _inside(self.a0[a], 2 - a)
            n = self.n[a]
            s.narrow(2 - a, 1, n - 1).sub_(inner * x.narrow(2 - a, 0, n - 1))
            s.narrow(2 - a, 0, n - 1).sub_(inner * x.narrow(2 - a, 1, n - 1))
        return torch.where(self.diag > 0, s, torch.zeros_like(s))

    def project(self, dt):
        dx, inv = self.dx, self.dx * self.dx / dt
        div = sum(self._hi(a, self.open[a] * self.vel[a]) - self._lo(a, self.open[a] * self.vel[a]) for a in range(3)) / dx
        b = (self.S - div) * inv
        for a in range(3):
            for side, at, view in ((0, 0, self._lo), (1, self.n[a] - 1, self._hi)):
                if a == 2 and side == 0:
                    continue
                v = view(a, self.vel[a]).select(2 - a, at)
                inflow = v < 0 if side else v > 0
                b.select(2 - a, at).add_(torch.where(inflow, -0.5 * v * v, torch.zeros_like(v)) *
                                         view(a, self.a0[a]).select(2 - a, at))
        b = torch.where(self.diag > 0, b, torch.zeros_like(b))
        x = torch.where(self.blocked, torch.zeros_like(b), self.f["p"])
        minv = torch.where(self.diag > 0, 1.0 / torch.clamp(self.diag, min=1e-300), torch.zeros_like(b))
        r = b - self._apply(x)
        z = minv * r
        d, rz, stop = z.clone(), (r * z).sum(), 1e-12 * b.abs().max()
        for it in range(6000):
            if it % 25 == 0 and bool(r.abs().max() <= stop):
                break
            q = self._apply(d)
            alpha = rz / (d * q).sum()
            x = x + alpha * d
            r = r - alpha * q
            z = minv * r
            rz, old = (r * z).sum(), rz
            d = z + (rz / old) * d
        self.f["p"] = x
        s = dt / dx
        self.max_vel = 0.0
        for a in range(3):
            dim, v, n = 2 - a, self.vel[a], self.n[a]
            hout = lambda u, inflow: torch.where(inflow, -0.5 * u * u, torch.zeros_like(u))
            hi = torch.cat([x, hout(v.narrow(dim, n, 1), v.narrow(dim, n, 1) < 0)], dim)
            lo = torch.cat([hout(v.narrow(dim, 0, 1), v.narrow(dim, 0, 1) > 0), x], dim)
            go = (self.am[a] > 0) & (self.open[a] > 0)
            if a < 2:
                for side in (0, 1):
                    if self.wind[a][side] is not None:
                        go.select(dim, n if side else 0).zero_()
            v = torch.where(go, torch.clamp(v - s * (hi - lo), -40.0, 40.0), v)
            v = torch.where(self.open[a] > 0, v, torch.zeros_like(v))
            self.vel[a] = v
            self.max_vel = max(self.max_vel, float((v.abs() * self.open[a]).max()))

    def advect(self, dt):
        dx, s = self.dx, dt / self.dx
        T, rho, gas = self.f["T"], self.rho(), ~self.blocked
        faces = []
        mden = rho
        solid = lambda a, by: _shift(self.blocked, 2 - a, by, False)

        def upwind(F, amb, a, by, un, inside, floor):
            """The neighbour's value, and the limited value carried through the face."""
            fn = _shift(F, 2 - a, by, amb)
            behind = torch.where(solid(a, -by), F, _shift(F, 2 - a, -by, amb))
            beyond = torch.where(solid(a, 2 * by), fn, _shift(F, 2 - a, 2 * by, amb))
            out = F + 0.5 * _superbee_times(F - behind, fn - F, floor)
            come = fn + 0.5 * _superbee_times(fn - beyond, F - fn, floor)
            return fn, torch.where(un > 0, out, come)

        for a, by, fo, inside, on in self.neighbours():
            un = by * fo * (self._hi if by > 0 else self._lo)(a, self.vel[a])
            _, tf = upwind(T, T0, a, by, un, inside, 1e-6)
            r_up = torch.where(on, self.P0 / (self.RS * torch.clamp(tf, min=200.0)), torch.zeros_like(tf))
            mden = mden - s * r_up * un
            nun = torch.where(inside, _shift(self.nu, 2 - a, by, 0.0), self.nu)
            Dd = 0.5 * (self.nu + nun) / 0.5 + 2.0e-5
            rfd = torch.where(inside, 0.5 * (rho + _shift(rho, 2 - a, by, 0.0)), rho)
            faces.append((a, by, fo, inside, on, un, r_up, Dd, rfd))
        for k in self.SCALARS:
            F, amb = self.f[k], self.AMB.get(k, 0.0)
            lo, hi, acc, macc = F, F, torch.zeros_like(F), torch.zeros_like(F)
            zero = torch.zeros_like(F)
            for a, by, fo, inside, on, un, r_up, Dd, rfd in faces:
                fn, face = upwind(F, amb, a, by, un, inside, 1e-12)
                lo = torch.where(on, torch.minimum(lo, fn), lo)
                hi = torch.where(on, torch.maximum(hi, fn), hi)
                move = -un * (face - F)
                carry = -r_up * un * face
                if k != "T":
                    move = move + fo * Dd * (fn - F) / dx
                    carry = carry + fo * rfd * Dd * (fn - F) / dx
                acc = acc + torch.where(on, move, zero)
                macc = macc + torch.where(on, carry, zero)
            value = torch.where(mden > 0.25 * rho, (rho * F + s * macc) / mden, F + s * acc)
            self.f[k] = torch.where(gas, torch.minimum(torch.maximum(value, lo), hi), F)
        self.time += dt

    def step(self, limit):
        dt = self.stable_dt(limit)
        self.combust(dt)
        self.turbulence()
        self.heat_and_energy(dt)
        self.momentum(dt)
        self.project(dt)
        self.advect(dt)
        return dt

    def fields(self):
        out = {k: v.reshape(-1).cpu().numpy() for k, v in zip("uvw", self.vel)}
        return out | {k: self.f[k].reshape(-1).cpu().numpy() for k in ("p",) + self.SCALARS}


def _trace64(c, w):
    """The radiation trace: four bands, 32 directions, a march of at most 8 m from every element."""
    dev, f64 = _device(), torch.float64
    t = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)
    pi, dx, n = 3.14159265, c.dx, (c.nx, c.ny, c.nz)
    N = c.N

    def below(lt):
        x = 14388.0 / lt
        s = 0.0
        for k in range(1, 13):
            s = s + torch.exp(-x * k) / k * (x**3 + 3 * x * x / k + 6 * x / (k * k) + 6.0 / (k**3))
        return torch.clamp(1.0 - 15.0 / pi**4 * s, 0.0, 1.0)

    def fractions(T):
        up = [below(e * T) for e in (2.7, 8.0, 14.0)]
        return torch.stack([up[0], up[1] - up[0], up[2] - up[1], 1.0 - up[2]], -1)

    f0 = fractions(t([T0]))[0]
    power = lambda T: 5.670374e-8 * (fractions(T) * (T**4)[..., None] - f0 * T0**4)
    i = torch.arange(32, dtype=f64, device=dev)
    z = 1.0 - 2.0 * (i + 0.5) / 32
    r = torch.sqrt(torch.clamp(1 - z * z, min=0.0))
    ang = pi * (3.0 - math.sqrt(5.0)) * i
    dirs = torch.stack([r * torch.cos(ang), r * torch.sin(ang), z], -1)
    dW = 4.0 * pi / 32
    blocked = t(c.blocked) > 0
    g = {k: t(v) for k, v in w["gas"].items()}
    T = torch.where(blocked, t(w["solidT"]), g["T"])
    E = power(T)
    rho = g["Pb"] / (287.0 * g["T"])
    pg = (g["Yw"] * 28.96 / 18.02 + g["Yc"] * 28.96 / 44.01) * g["Pb"] / 101325.0
    kap = 5.5 * (rho * g["Ys"] / 1800.0)[:, None] / (t([1.5, 4.5, 11.0, 25.0]) * 1e-6) + t([0.05, 3.0, 0.1, 6.0]) * pg[:, None] + 1e-4
    jf = torch.where(g["hrr"] > 0, 0.35 * g["hrr"] / (4.0 * pi), torch.zeros_like(rho))
    j = kap * E / pi
    flame = (jf > j.sum(-1)) & ~blocked
    j = torch.where(flame[:, None], jf[:, None] * fractions(t([1400.0]))[0], j)
    src = torch.where(blocked[:, None], E * (0.9 / pi), j / kap)
    nf = ((c.nx + 1) * c.ny * c.nz, c.nx * (c.ny + 1) * c.nz)
    wl = np.asarray(w["walls"], np.float64).reshape(-1, 4)
    wall_of = torch.full((nf[0] + nf[1] + c.nx * c.ny * (c.nz + 1),), -1, dtype=torch.int64, device=dev)
    off = np.array([0, nf[0], nf[0] + nf[1]])
    if len(wl):
        wall_of[torch.tensor(off[wl[:, 0].astype(int)] + wl[:, 1].astype(np.int64), device=dev)] = torch.arange(len(wl), device=dev)
        wall_i = torch.stack([power(t(wl[:, 2])), power(t(wl[:, 3]))], 1) * (0.9 / pi)
    el = t(w["elements"])
    cos = el[:, 3:6] @ dirs.T
    sphere = el[:, 9:10] > 0
    norm = pi / torch.clamp((torch.clamp(cos, min=0.0) * dW).sum(-1, keepdim=True), min=1e-300)
    weight = torch.where(sphere, dW * 0.25 * el[:, 6:7], cos * dW * norm * el[:, 6:7])
    org = (el[:, 0:3] - t([c.ox, c.oy, c.oz])) / dx
    cell0 = torch.floor(org).long()
    lim = torch.tensor(n, device=dev)
    valid = ((cell0 >= 0) & (cell0 < lim)).all(-1, keepdim=True) & (sphere | (cos > 0))
    Is = el[:, 7:8] / pi * power(el[:, 8])
    absorbed = torch.zeros(len(el), dtype=f64, device=dev)
    gas = torch.zeros(N, dtype=f64, device=dev)
    ids = valid.nonzero()
    for part in ids.split(1 << 21):
        e, d = part[:, 0], part[:, 1]
        dv, p, cell = dirs[d], org[e], cell0[e].clone()
        sign = torch.where(dv > 1e-9, 1, torch.where(dv < -1e-9, -1, 0))
        far = torch.full_like(dv, 1e30)
        tm = torch.where(sign > 0, (cell + 1 - p) / dv, torch.where(sign < 0, (p - cell) / -dv, far))
        td = torch.where(sign == 0, far, 1 / dv.abs().clamp(min=1e-9))
        eps, wt = el[e, 7], weight[e, d]
        skip = torch.where(el[e, 10] > 0, cell[:, 0] + c.nx * (cell[:, 1] + c.ny * cell[:, 2]), -1)
        tau, I, now = torch.ones(len(e), 4, dtype=f64, device=dev), torch.zeros(len(e), 4, dtype=f64, device=dev), torch.zeros(len(e), dtype=f64, device=dev)
        end, ise, own = torch.zeros_like(I), Is[e], e
        while len(e):
            a = torch.where(tm[:, 0] < tm[:, 1], torch.where(tm[:, 0] < tm[:, 2], 0, 2), torch.where(tm[:, 1] < tm[:, 2], 1, 2))
            tn = torch.clamp(tm.gather(1, a[:, None])[:, 0], max=8.0 / dx)
            ds = (tn - now) * dx
            cid = cell[:, 0] + c.nx * (cell[:, 1] + c.ny * cell[:, 2])
            on = (ds > 0) & ~blocked[cid] & (cid != skip)
            x = kap[cid] * ds[:, None]
            att = torch.where(x < 1e-3, x * (1 - 0.5 * x), 1.0 - torch.exp(-x))
            got = tau * src[cid] * att
            gain = (ise * tau * att - torch.where(flame[cid][:, None], torch.zeros_like(got), eps[:, None] * got)).sum(-1)
            gas.index_add_(0, cid, torch.where(on, wt * gain, torch.zeros_like(gain)))
            I = torch.where(on[:, None], I + got, I)
            tau = torch.where(on[:, None], tau * (1.0 - att), tau)
            now = tn
            done = (now >= 8.0 / dx) | (tau < 1e-3).all(-1)
            st = sign.gather(1, a[:, None])[:, 0]
            up = (st > 0).long()
            q = [cell[:, m] + (a == m) * up for m in range(3)]
            face = torch.where(a == 0, q[0] + (c.nx + 1) * (q[1] + c.ny * q[2]),
                               torch.where(a == 1, nf[0] + q[0] + c.nx * (q[1] + (c.ny + 1) * q[2]),
                                           nf[0] + nf[1] + q[0] + c.nx * (q[1] + c.ny * q[2])))
            wall = wall_of[face]
            hit = ~done & (wall >= 0)
            if len(wl):
                end = torch.where(hit[:, None], wall_i[wall.clamp(min=0), 1 - up], end)
            done = done | hit
            cell = cell + torch.nn.functional.one_hot(a, 3) * st[:, None]
            out = ((cell < 0) | (cell >= lim)).any(-1)
            done = done | out
            nid = torch.where(done, 0, cell[:, 0] + c.nx * (cell[:, 1] + c.ny * cell[:, 2]))
            stop = ~done & blocked[nid]
            end = torch.where(stop[:, None], src[nid], end)
            done = done | stop
            tm = tm + torch.nn.functional.one_hot(a, 3) * td
            if bool(done.any()):
                value = (I + tau * end).sum(-1) * eps * wt
                absorbed.index_add_(0, own[done], value[done])
                go = ~done
                e, dv, cell, sign, tm, td, eps, wt, skip, tau, I, now, end, ise, own = (
                    v[go] for v in (e, dv, cell, sign, tm, td, eps, wt, skip, tau, I, now, end, ise, own))
    return {"absorbed": absorbed.cpu().numpy(), "gas": gas.cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "render":
        return None
    cs = _buildings(case)
    if case["kind"] == "rad":
        return _trace64(cs[0], _trace_inputs(cs[0], case, seed))
    # steps x buildings at 20 ms or more each: a large batch would take minutes
    if len(cs) * case["steps"] > 200:
        return None
    limits = _step_limits(len(cs)) if case["kind"] == "batch" else [DT_MAX]
    dts, fields = [], []
    for c, limit in zip(cs, limits):
        state, time = _fire_state(c, seed)
        room = _Room64(c, state, time, max(float(np.abs(state[f]).max()) for f in "uvw"))
        if not room.open_zones_only():
            return None
        dts.append([room.step(float(limit)) for _ in range(case["steps"])])
        fields.append(room.fields())
    dt = np.array(dts).T
    out = {"dt": dt if case["kind"] == "batch" else dt[:, 0]}
    return out | {f: np.concatenate([x[f] for x in fields]) for f in STATE}
