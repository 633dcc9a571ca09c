"""Performance cases of the room solver: what its users run, through its public entry points.

    fluid   one projection room stepped through ``FluidHandle`` (FP64 plain CG as ff-room's own
            scenes run it, or mixed precision with the multigrid solve and the schedule the
            server gives a room of that size)
    batch   many uneven rooms stepped together (``BatchHandle``)
    solve   one request from host buffers and back: create, step, read every field, close
    lbm     one D3Q19 room (``LbmHandle``) in FP64, FP32 or FP16 population storage

Rooms come from ``SceneConfig`` as a user writes one: a few wall fans, boxes on the floor, the
automatic outflow wall or a window with an outside temperature, a heated floor.  A projection
room starts from a smooth velocity field (a run taken up again), an LBM room after ten steps.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ff-room_b200"))

from ffrb import capi, workloads  # noqa: E402
from ffrb.params import params_from_scene  # noqa: E402
from ffrb.scene import (FanConfig, HeatPatchConfig, ObstacleConfig, OpeningConfig, RoomConfig,  # noqa: E402
                        SceneConfig, SolverConfig, build_room)
from ffrb.serve import Schedule, Tuner, apply_schedule  # noqa: E402

LBM_SPIN_UP = 10
EXACT_CELLS = 2_000_000     # above this the 64-bit projection takes minutes


def _fluid(name, grid, precision, steps, scheme="upwind", heat=False, window=False, tol=1e-6, stretch=1.0):
    return {"name": name, "kind": "fluid", "nx": grid[0], "ny": grid[1], "nz": grid[2], "precision": precision,
            "steps": steps, "scheme": scheme, "heat": heat, "window": window, "tol": tol, "stretch": stretch}


def _lbm(name, grid, storage, steps):
    return {"name": name, "kind": "lbm", "nx": grid[0], "ny": grid[1], "nz": grid[2], "storage": storage,
            "steps": steps}


def listed():
    return [
        # the example scene's grid under the LBM method, one step per call: what run_animated and
        # every per-step callback pay
        _lbm("lbm_example_fp64", (25, 20, 12), "fp64", 1),
        # the same scene under the projection method in the reference's FP64, one step per call
        _fluid("room_example_fp64", (25, 20, 12), "fp64", 1),
        # a summer-cooling scene: windows, buoyancy, QUICK on an odd grid, a few steps per call
        _fluid("room_window_quick_fp64", (41, 33, 19), "fp64", 3, "quick", heat=True, window=True),
        # the thermal room at the resolution its 2000-step reference run has, FP64 plain CG
        _fluid("room_thermal_fp64", (80, 64, 24), "fp64", 1, heat=True, tol=1e-8),
        # a small and a medium request of the serving stream, stepped as the server steps them
        _fluid("request_small_mixed", (48, 40, 27), "mixed", 10, heat=True),
        _fluid("request_odd_mixed", (161, 127, 49), "mixed", 3, heat=True),
        # the large thermal room of the headline benchmark
        _fluid("room_large_mixed", (320, 256, 96), "mixed", 2, heat=True, tol=1e-8),
        # uneven rooms advanced in one batch
        {"name": "batch_uneven_mixed", "kind": "batch", "rooms": 12, "low": 32, "high": 96, "steps": 3},
        # one request end to end: host room in, host fields out
        {"name": "solve_from_host_mixed", "kind": "solve", "nx": 96, "ny": 80, "nz": 41, "steps": 20},
        # LBM rooms in each storage: medium and ragged, then the benchmark lattice
        _lbm("lbm_medium_fp64", (130, 97, 65), "fp64", 4),
        _lbm("lbm_ragged_fp16", (301, 203, 101), "fp16", 3),
        _lbm("lbm_large_fp32", (384, 320, 128), "fp32", 2),
    ]


def _draw_grid(rng, low, high):
    """A room of about log-uniform size in [low, high] cells, each axis at least 8."""
    cells = math.exp(rng.uniform(math.log(low), math.log(high)))
    shape = [rng.uniform(1.0, 2.5), rng.uniform(1.0, 2.5), rng.uniform(0.6, 1.2)]
    h = (cells / (shape[0] * shape[1] * shape[2])) ** (1.0 / 3.0)
    return [max(8, int(round(s * h))) for s in shape]


def draw(rng):
    kind = rng.choice(["fp64", "mixed", "mixed", "batch", "solve", "lbm", "lbm"])
    if kind == "lbm":
        g = _draw_grid(rng, 6_000, 8_000_000)
        small = g[0] * g[1] * g[2] < 3_000_000
        case = _lbm("", g, rng.choice(["fp64", "fp32", "fp16"]), rng.randint(1, 4) if small else 1)
    elif kind == "batch":
        case = {"kind": "batch", "rooms": rng.randint(3, 14), "low": 32, "high": rng.randint(48, 96),
                "steps": rng.randint(1, 4)}
    elif kind == "solve":
        g = _draw_grid(rng, 15_000, 500_000)
        case = {"kind": "solve", "nx": g[0], "ny": g[1], "nz": g[2], "steps": rng.randint(5, 20)}
    else:
        fp64 = kind == "fp64"
        # (plain CG is left to uniform grids, where its operator is symmetric on the fluid cells)
        case = _fluid("", _draw_grid(rng, 6_000 if fp64 else 14_000, 110_000 if fp64 else 4_000_000), kind,
                      rng.randint(1, 3), rng.choice(["upwind", "upwind", "quick"]),
                      heat=rng.random() < 0.6, window=rng.random() < 0.25, tol=rng.choice([1e-6, 1e-6, 1e-8]),
                      stretch=1.0 if fp64 else rng.choice([1.0, 1.0, 1.0, 1.02]))
    case.pop("name", None)
    return case


# ------------------------------------------------------------------ inputs

def _scene(case, seed):
    rng = np.random.default_rng(seed)
    grid = (case["nx"], case["ny"], case["nz"])
    h = (96.0 / (grid[0] * grid[1] * grid[2])) ** (1.0 / 3.0)     # a room of about 96 m^3
    size = tuple(n * h for n in grid)
    lx, ly, lz = size
    rad = max(0.2, 1.1 * h)
    fans = [FanConfig((0.08 * lx, float(rng.uniform(0.3, 0.7)) * ly, float(rng.uniform(0.35, 0.65)) * lz),
                      (0.0, 0.0), float(rng.uniform(2.0, 4.0)), rad, "west"),
            FanConfig((float(rng.uniform(0.3, 0.7)) * lx, 0.08 * ly, float(rng.uniform(0.35, 0.65)) * lz),
                      (90.0, 0.0), float(rng.uniform(1.0, 3.0)), rad, "south")]
    boxes = []
    for b in range(3):
        x0, y0 = float(rng.uniform(0.15, 0.7)) * lx, float(rng.uniform(0.15, 0.7)) * ly
        boxes.append(ObstacleConfig((x0, y0, 0.0), (x0 + 0.15 * lx, y0 + 0.15 * ly,
                                                    float(rng.uniform(0.2, 0.5)) * lz), f"box{b}"))
    mixed = case["kind"] == "solve" or case.get("precision") == "mixed"
    heat, window = bool(case.get("heat", case["kind"] == "solve")), bool(case.get("window"))
    cfg = SceneConfig(
        room=RoomConfig(size, grid, float(case.get("stretch", 1.0))), fans=fans, obstacles=boxes,
        openings=[OpeningConfig("east", (0.5 * ly, 0.5 * lz), (0.4 * ly, 0.4 * lz), 32.0),
                  OpeningConfig("north", (0.6 * lx, 0.5 * lz), (0.2 * lx, 0.3 * lz), 30.0)] if window else [],
        heat_patches=[HeatPatchConfig("floor", (0.3 * lx, 0.7 * lx), (0.3 * ly, 0.7 * ly), 25.0),
                      HeatPatchConfig("ceiling", (0.3 * lx, 0.7 * lx), (0.3 * ly, 0.7 * ly), 18.0)] if heat else [],
        solver=SolverConfig(max_steps=100000, convergence_tol=1e-4, poisson_max_iter=2000,
                            poisson_tol=float(case.get("tol", 1e-6)), advection=case.get("scheme", "upwind"),
                            buoyancy=heat or window, precision="mixed" if mixed else "fp64",
                            poisson_method="multigrid" if mixed else "cg"))
    # QUICK with explicit Euler steps needs the smaller Courant number to stay bounded over long runs
    cfg.solver.dt = workloads.room_dt(cfg, 0.1 if case.get("scheme") == "quick" else 0.5)
    return cfg


def _flow(room, seed):
    """A smooth velocity field of about 0.5 m/s with no flow through the walls."""
    rng = np.random.default_rng([seed, 1])
    faces = [room.xs / room.lx, room.ys / room.ly, room.zs / room.lz]
    centres = [0.5 * (f[1:] + f[:-1]) for f in faces]
    init = {}
    for axis, name in enumerate("uvw"):
        total = 0.0
        for _ in range(3):
            modes = rng.integers(1, 5, 3)
            parts = [np.sin(np.pi * modes[a] * faces[a]) if a == axis else np.cos(np.pi * modes[a] * centres[a])
                     for a in range(3)]
            total = total + (float(rng.uniform(-0.3, 0.3)) * parts[0][:, None, None] * parts[1][None, :, None]
                             * parts[2][None, None, :])
        init[name] = total.reshape(-1)
    return init


def _serving_table():
    import json
    with open(os.path.join("ff-room_b200", "ffrb", "tuned_b200.json")) as fh:
        return Tuner.from_json(json.load(fh)["table"])


def _batch_rooms(case, seed):
    """The batch's rooms: uneven sizes that the case fixes, the scenes from the seed."""
    dims = np.random.default_rng(7).integers(case["low"], case["high"] + 1, (case["rooms"], 3))
    out = []
    for i, (nx, ny, nz) in enumerate(dims):
        cfg = _scene({"kind": "batch", "nx": int(nx), "ny": int(ny), "nz": int(nz), "precision": "mixed"},
                     100 * seed + i)
        room = build_room(cfg)
        out.append((room, params_from_scene(cfg), _flow(room, 100 * seed + i)))
    return out


def _lbm_room(case, seed):
    cfg = _scene(case, seed)
    room = build_room(cfg)
    speed = max(f.velocity for f in cfg.fans)
    return room, 0.8, 0.05 * room.dx / speed        # fan at lattice speed 0.05


def _view(handle, name):
    """A field of the handle as a tensor, without a copy; the tensor keeps the handle alive."""
    array = capi.DeviceArray(handle.field_dev(name), int(np.prod(handle.room.shapes()[name])))
    array.owner = handle
    return torch.as_tensor(array, device="cuda")


def _views(handle, names):
    return {k: _view(handle, k) for k in names}


def prepare(case, seed):
    torch.cuda.init()
    kind = case["kind"]
    state = {"case": case}
    if kind == "lbm":
        room, tau, dt = _lbm_room(case, seed)
        h = capi.LbmHandle(room, tau, 100000, 1e-4, dt, case["storage"])
        h.advance(LBM_SPIN_UP)
        state.update(handle=h, fields=_views(h, "uvwp"))
    elif kind == "batch":
        handles = []
        for room, params, init in _batch_rooms(case, seed):
            h = capi.FluidHandle(room, params, init)
            apply_schedule(h, Schedule(0, 20, False, 16), room, params)     # one cluster per room
            handles.append(h)
        batch = capi.BatchHandle(handles)
        batch.use_graph(True)
        state.update(batch=batch, handles=handles, fields=[_views(h, "uvwp") for h in handles])
    else:
        cfg = _scene(case, seed)
        room, params = build_room(cfg), params_from_scene(cfg)
        init = _flow(room, seed)
        state.update(room=room, params=params, init=init, schedule=_serving_table().schedule(room))
        if kind == "fluid":
            h = capi.FluidHandle(room, params, init)
            if case["precision"] == "mixed":
                apply_schedule(h, state["schedule"], room, params)
            h.synchronize()
            state.update(handle=h, fields=_views(h, "uvwp"), init=None)
    return state


# --------------------------------------------------------------------- run

def _history(records, keys):
    """Step results by name.  What a pressure solve leaves behind (its residual, the largest
    divergence) is rounding on top of its stopping error and is no result of the step."""
    return {k: np.array([r[k] for r in records]) for k in keys}


FLUID_KEYS = ("step", "velocity_change", "converged", "T_mean", "cg_iterations", "flags")
LBM_KEYS = ("step", "velocity_change", "divergence_max", "converged", "flags")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "lbm":
        h = state["handle"]
        records = [h.step()] if case["steps"] == 1 else h.advance(case["steps"])
        return {**state["fields"], **_history(records, LBM_KEYS)}
    if kind == "fluid":
        h = state["handle"]
        records = [h.step()] if case["steps"] == 1 else h.advance(case["steps"])
        out = {**state["fields"], **_history(records, FLUID_KEYS)}
        if state["params"].thermal:
            out["T"] = _view(h, "T")      # the solver swaps this buffer
        return out
    if kind == "batch":
        records = state["batch"].advance(case["steps"])
        return {"rooms": state["fields"],
                **{k: np.array([[r[k] for r in room] for room in records])
                   for k in ("velocity_change", "converged", "cg_iterations", "flags")}}
    h = capi.FluidHandle(state["room"], state["params"], state["init"])
    apply_schedule(h, state["schedule"], state["room"], state["params"])
    records = h.advance(case["steps"])
    out = {k: h.get(k) for k in "uvwpT"}
    h.close()
    return {**out, **_history(records, FLUID_KEYS)}


# -------------------------------------------------------------------- work

def work(case):
    """Per step: every field read once and written once, the cell types read once."""
    kind = case["kind"]
    if kind == "batch":
        cells = case["rooms"] * (0.5 * (case["low"] + case["high"])) ** 3
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    steps = case["steps"]
    if kind == "lbm":
        size = {"fp64": 8, "fp32": 4, "fp16": 2}[case["storage"]]
        # populations in and out, new faces and pressure out, old faces in (max |du|)
        return {"bytes": steps * cells * (2 * 19 * size + 32 + 24 + 1), "flops": steps * cells * 350}
    thermal = case.get("heat", kind == "solve") or case.get("window")
    fields = 5 if thermal else 4
    bytes_ = steps * cells * (2 * 8 * fields + 1)
    if kind == "solve":
        bytes_ += cells * (3 * 8 + 1 + 5 * 8)       # the request in, the fields out
    return {"bytes": bytes_, "flops": steps * cells * 500}


# ------------------------------------------------------------------- exact
#
# The same steps in plain torch, 64 bits, with the pressure equation solved to rounding.

def _shift(a, axis, by, fill=0.0):
    """b[i] = a[i - by] along axis; `fill` (a number, or values of a's shape) where that is outside."""
    b = torch.roll(a, by, axis)
    n = a.shape[axis]
    edge = slice(0, by) if by > 0 else slice(n + by, n)
    at = tuple(edge if d == axis else slice(None) for d in range(3))
    b[at] = fill if isinstance(fill, float) else fill[at]
    return b


def _along(v, axis):
    return v.reshape([-1 if a == axis else 1 for a in range(3)])


def _advect(scheme, mm, m, c, p, a, h, quick):
    """Flux difference along one axis; `quick` is the mask of the faces where QUICK is active."""
    up = torch.where(a > 0, a * (c - m) / h, a * (p - c) / h)
    if scheme != "quick":
        return up
    pos = (6 * c + 3 * p - m) / 8 - (6 * m + 3 * c - mm) / 8
    neg = (6 * p + 3 * c - mm) / 8 - (6 * c + 3 * p - m) / 8
    return torch.where(quick, a * torch.where(a >= 0, pos, neg) / h, up)


class _ExactRoom:
    def __init__(self, room, params):
        dev = "cuda"
        self.room, self.prm = room, params
        self.n = (room.nx, room.ny, room.nz)
        self.ct = torch.tensor(room.cell_type.astype(np.int64), device=dev).reshape(self.n)
        self.h = [torch.tensor(np.asarray(v), dtype=torch.float64, device=dev) for v in (room.dxv, room.dyv, room.dzv)]
        self.hb = [_along(h, a) for a, h in enumerate(self.h)]
        self.scheme = ("upwind", "quick")[params.advection]
        self.solid = self.ct == 1
        self.active = (self.ct == 0) | (self.ct == 2)
        self.out = self.ct == 3
        self._pressure_rows()

    def _index(self, shape, axis):
        return _along(torch.arange(shape[axis], device="cuda"), axis)

    def quick_mask(self, shape, own=None):
        ok = torch.ones(shape, dtype=torch.bool, device="cuda")
        for a in range(3):
            i = self._index(shape, a)
            ok = ok & (i >= (2 if a == own else 1)) & (i <= self.n[a] - 2)
        return ok

    def _pressure_rows(self):
        """Weights 1 / (face distance * width) to each neighbour and what the neighbour is."""
        self.rows = []
        diag = torch.zeros(self.n, dtype=torch.float64, device="cuda")
        for a in range(3):
            h = self.h[a]
            dist = 0.5 * (h[1:] + h[:-1])
            for by, d in ((1, torch.cat([h[:1], dist])), (-1, torch.cat([dist, h[-1:]]))):
                s = _along(1.0 / (d * h), a).expand(self.n)
                nb_active = _shift(self.active.double(), a, by) > 0
                nb_out = _shift(self.out.double(), a, by) > 0
                diag = diag + torch.where(nb_active, s, torch.where(nb_out, 2 * s, torch.zeros_like(s)))
                self.rows.append((a, by, torch.where(nb_active, s, torch.zeros_like(s))))
        self.diag = torch.where(diag > 1e-30, diag, torch.ones_like(diag))
        self.vol = (self.hb[0] * self.hb[1] * self.hb[2]).expand(self.n)

    def _couple(self, x):
        return sum(s * _shift(x, a, by) for a, by, s in self.rows)

    def pressure(self, b):
        """Conjugate gradients on the volume-scaled fluid rows, then the outflow rows."""
        act = self.active.double()
        inv = act / (self.diag * self.vol)
        r = b * self.vol * act
        x = torch.zeros_like(r)
        goal = 1e-12 * float(r.norm())
        z = inv * r
        d = z.clone()
        rz = (r * z).sum()
        for it in range(20000):
            if it % 50 == 0 and float(r.norm()) <= goal:
                break
            q = (self.diag * d - self._couple(d)) * self.vol * act
            alpha = rz / (d * q).sum()
            x += alpha * d
            r -= alpha * q
            z = inv * r
            new = (r * z).sum()
            d = z + (new / rz) * d
            rz = new
        return torch.where(self.out, (b + self._couple(x)) / self.diag, x)

    def predict(self, vel, T):
        prm, out = self.prm, []
        for d in range(3):
            f = vel[d]
            own = self._index(f.shape, d)
            inner = (own > 0) & (own < self.n[d])
            quick = self.quick_mask(f.shape, d)
            adv = dif = 0.0
            for a in range(3):
                m, p = _shift(f, a, 1), _shift(f, a, -1)
                if a == d:      # the wall's own face reads as zero
                    m, p = m * (own > 1), p * (own < self.n[d] - 1)
                    speed, h = f, _along(torch.cat([self.h[a], self.h[a][-1:]]), a)
                else:
                    g = vel[a].narrow(a, 0, self.n[a])
                    pad = g.narrow(d, self.n[d] - 1, 1)
                    g = torch.cat([g, pad], d)
                    speed = 0.5 * (_shift(g, d, 1) + g) * (self._index(f.shape, a) > 0)
                    h = self.hb[a]
                mm = m
                if self.scheme == "quick" and (d == 0 or a == d):   # by flat index, across rows too
                    stride = f.stride(a)
                    mm = torch.roll(f.reshape(-1), 2 * stride).reshape(f.shape)
                adv = adv + _advect(self.scheme, mm, m, f, p, speed, h, quick)
                dif = dif + (m - 2 * f + p) / (h * h)
            new = torch.where(inner, f + prm.dt * (prm.nu * dif - adv), f)
            if d == 2 and prm.buoyancy:
                new[:, :, 1:-1] += prm.g_accel * prm.beta * prm.dt * (0.5 * (T[:, :, :-1] + T[:, :, 1:])
                                                                      - prm.T_initial)
            out.append(new)
        return out

    def boundary(self, vel):
        for a in range(3):
            f, n = vel[a], self.n[a]
            for face, cell in ((0, 0), (n, n - 1)):
                keep = self.out.select(a, cell)
                f.select(a, face)[~keep] = 0.0
            f.narrow(a, 0, n)[self.solid] = 0.0
            f.narrow(a, 1, n)[self.solid] = 0.0
        for fan in self.room.fans:
            i0, i1, j0, j1, k0, k1 = fan.box
            lo, hi = (i0, j0, k0), (i1, j1, k1)
            for a in range(3):
                if fan.vel[a] != 0.0:
                    at = tuple(slice(max(0, lo[e]), min(self.n[e] - 1, hi[e]) + 1 + (e == a)) for e in range(3))
                    vel[a][at] = fan.vel[a]

    def _patch(self, p, inner):
        """Index of a patch's cells in the wall layer, or in the layer `inner` cells in."""
        at = [slice(p.a_min, p.a_max + 1), slice(p.b_min, p.b_max + 1)]
        at.insert(p.axis, self.n[p.axis] - 1 - inner if p.side else inner)
        return tuple(at)

    def opening_temperature(self, vel, T):
        for p in self.room.openings:
            face = list(self._patch(p, 0))
            face[p.axis] = self.n[p.axis] if p.side else 0
            v = vel[p.axis][tuple(face)]
            enters = (v <= 0) if p.side else (v >= 0)
            T[self._patch(p, 0)] = torch.where(enters, torch.full_like(v, p.T_outside), T[self._patch(p, 1)])

    def temperature(self, vel, T):
        prm = self.prm
        quick = self.quick_mask(self.n)
        fluid = self.ct == 0
        adv = dif = 0.0
        for a in range(3):
            def at(by):
                v = _shift(T, a, by, T)
                return torch.where(_shift(self.solid.double(), a, by) > 0, T, v)
            m, p, mm = at(1), at(-1), at(2)
            speed = 0.5 * (vel[a].narrow(a, 0, self.n[a]) + vel[a].narrow(a, 1, self.n[a]))
            adv = adv + _advect(self.scheme, mm, m, T, p, speed, self.hb[a], quick)
            dif = dif + (m - 2 * T + p) / (self.hb[a] * self.hb[a])
        new = T + prm.dt * (prm.k_thermal / (prm.rho * prm.cp) * dif - adv)
        return torch.where(fluid, new, T)

    def steps(self, init, count):
        prm, n = self.prm, self.n
        vel = [torch.tensor(np.asarray(init[k]), dtype=torch.float64, device="cuda").reshape(self.room.shapes()[k])
               for k in "uvw"]
        T = torch.full(n, float(prm.T_initial), dtype=torch.float64, device="cuda")
        if prm.thermal:
            self.opening_temperature(vel, T)
        change, mean = [], []
        for _ in range(count):
            old = [f.clone() for f in vel]
            vel = self.predict(vel, T)
            self.boundary(vel)
            div = sum((vel[a].narrow(a, 1, n[a]) - vel[a].narrow(a, 0, n[a])) / self.hb[a] for a in range(3))
            P = self.pressure(torch.where(self.solid, torch.zeros_like(div), -(prm.rho / prm.dt) * div))
            for a in range(3):
                dist = _along(0.5 * (self.h[a][1:] + self.h[a][:-1]), a)
                vel[a].narrow(a, 1, n[a] - 1).sub_(prm.dt / prm.rho * torch.diff(P, dim=a) / dist)
            self.boundary(vel)
            for p in self.room.outflows:
                to, source = list(self._patch(p, 0)), list(self._patch(p, 0))
                to[p.axis] = n[p.axis] if p.side else 0
                source[p.axis] = n[p.axis] - 1 if p.side else 1
                vel[p.axis][tuple(to)] = vel[p.axis][tuple(source)]
            if prm.thermal:
                self.opening_temperature(vel, T)
                T = self.temperature(vel, T)
                self.opening_temperature(vel, T)
                mean.append(float(T[self.ct == 0].mean()))
            else:
                mean.append(float(prm.T_initial))
            change.append(max(float((f - o).abs().max()) for f, o in zip(vel, old)) / prm.dt)
            for hp in self.room.heats:
                i0, i1, j0, j1, k0, k1 = hp.box
                T[i0:i1 + 1, j0:j1 + 1, k0:k1 + 1] = hp.T
        out = {k: f.reshape(-1) for k, f in zip("uvw", vel)}
        out.update(p=P.reshape(-1), T=T.reshape(-1), velocity_change=np.array(change), T_mean=np.array(mean))
        return out


def _d3q19():
    e = [(0, 0, 0)]
    for a in range(3):
        e += [tuple(s if d == a else 0 for d in range(3)) for s in (1, -1)]
    for a, b in ((0, 1), (0, 2), (1, 2)):
        e += [tuple(s if d == a else t if d == b else 0 for d in range(3)) for t in (1, -1) for s in (1, -1)]
    return e, [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12


def _exact_lbm(case, seed):
    room, tau, dt = _lbm_room(case, seed)
    n = (room.nx, room.ny, room.nz)
    e, w = _d3q19()
    mirror = [0] + [q + 1 if q % 2 else q - 1 for q in range(1, 19)]    # the solver's bounce-back pairs
    ct = torch.tensor(room.cell_type.astype(np.int64), device="cuda").reshape(n)
    open_ = ct != 1
    to_lattice, to_metres = dt / room.dx, room.dx / dt

    def moved(a, q, fill):
        for axis in range(3):
            if e[q][axis]:
                a = _shift(a, axis, e[q][axis], fill)
        return a

    def equilibrium(q, rho, u):
        eu = sum(float(e[q][a]) * u[a] for a in range(3) if e[q][a]) if q else torch.zeros_like(u[0])
        return w[q] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * sum(x * x for x in u))

    def moments(f):
        rho = sum(f)
        safe = torch.where(rho > 1e-14, rho, torch.ones_like(rho))
        return rho, [sum(float(e[q][a]) * f[q] for q in range(19) if e[q][a]) / safe for a in range(3)]

    def inflow(f):
        for fan in room.fans:
            i0, i1, j0, j1, k0, k1 = (max(0, b) for b in fan.box)
            at = (slice(i0, i1 + 1), slice(j0, j1 + 1), slice(k0, k1 + 1))
            here = ct[at] == 2
            u = [torch.tensor(v * to_lattice, dtype=torch.float64, device="cuda") for v in fan.vel]
            for q in range(19):
                f[q][at][here] = equilibrium(q, 1.0, u)

    def blocked(q):
        """Cells from which direction q leads out of the room or into a solid."""
        back = e.index(tuple(-x for x in e[q]))
        return moved(open_.double(), back, 0.0) == 0

    f = [torch.full(n, w[q], dtype=torch.float64, device="cuda") for q in range(19)]
    faces = [torch.zeros([m + (d == a) for d, m in enumerate(n)], dtype=torch.float64, device="cuda")
             for a in range(3)]
    P = torch.zeros(n, dtype=torch.float64, device="cuda")
    change, worst = [], []
    for _ in range(LBM_SPIN_UP + case["steps"]):
        inflow(f)
        rho, u = moments(f)
        collide = (ct == 0) | (ct == 3)
        for q in range(19):
            f[q] = torch.where(collide, f[q] + (equilibrium(q, rho, u) - f[q]) / tau, f[q])
        g = [torch.zeros_like(P) for _ in range(19)]
        for q in range(19):
            stop = blocked(q)
            g[mirror[q]] += torch.where(open_ & stop, f[q], torch.zeros_like(P))
            g[q] += moved(torch.where(open_ & ~stop, f[q], torch.zeros_like(P)), q, 0.0)
        f = g
        for p in room.outflows:
            to = [slice(p.a_min, p.a_max + 1), slice(p.b_min, p.b_max + 1)]
            source = list(to)
            to.insert(p.axis, n[p.axis] - 1 if p.side else 0)
            source.insert(p.axis, n[p.axis] - 2 if p.side else 1)
            here = ct[tuple(to)] == 3
            for q in range(19):
                f[q][tuple(to)] = torch.where(here, f[q][tuple(source)], f[q][tuple(to)])
        rho, u = moments(f)
        P = torch.where(open_, rho / 3, P)
        new = []
        for a in range(3):
            c = torch.where(open_, u[a] * to_metres, torch.zeros_like(P))
            mid = 0.5 * (c.narrow(a, 0, n[a] - 1) + c.narrow(a, 1, n[a] - 1))
            new.append(torch.cat([c.narrow(a, 0, 1), mid, c.narrow(a, n[a] - 1, 1)], a))
        change.append(max(float((x - y).abs().max()) for x, y in zip(new, faces)) / dt)
        faces = new
        h = [_along(torch.tensor(np.asarray(v), dtype=torch.float64, device="cuda"), a)
             for a, v in enumerate((room.dxv, room.dyv, room.dzv))]
        div = sum(torch.diff(x, dim=a) / h[a] for a, x in enumerate(faces))
        worst.append(float(div[ct == 0].abs().max()))
    k = case["steps"]
    return {**{name: x.reshape(-1) for name, x in zip("uvw", faces)}, "p": P.reshape(-1), "step": None,
            "velocity_change": np.array(change[-k:]), "divergence_max": np.array(worst[-k:]), "converged": None,
            "flags": None}


def exact(case, seed):
    if case["kind"] == "lbm":
        return _exact_lbm(case, seed)
    whole = {"step": None, "converged": None, "cg_iterations": None, "flags": None}
    if case["kind"] == "batch":
        rooms = [_ExactRoom(room, params).steps(init, case["steps"])
                 for room, params, init in _batch_rooms(case, seed)]
        return {"rooms": [{k: r[k] for k in "uvwp"} for r in rooms], "converged": None, "cg_iterations": None,
                "flags": None, "velocity_change": np.array([r["velocity_change"] for r in rooms])}
    if case["nx"] * case["ny"] * case["nz"] > EXACT_CELLS:
        return None
    cfg = _scene(case, seed)
    room, params = build_room(cfg), params_from_scene(cfg)
    out = _ExactRoom(room, params).steps(_flow(room, seed), case["steps"])
    if not params.thermal:
        out.pop("T")
    return {**out, **whole}
