"""Work that programs on this framework have it do, for timing and for comparing results.

Every case is a pass through the public entry points: the substeps of one output frame of a coupled or air-only
simulation (``HeatflowMPM``), a batch of uneven scenes (``AirBatch``), a served list of requests (``AirServer``), or a
the inside test that fills a mesh with particles (``winding_inside``).  Inputs come from the seed: a smooth solenoidal
velocity field, a warm plume and, in coupled scenes, a jittered particle body on the floor, sixteen substeps on (advanced
in plain torch, so that the fan's start is over and the pressure is the warm start that a running simulation has).
Passes of more than one substep begin from the same state each time, as a program does that goes back to a saved one; a
single substep simply goes on.  Batches and served requests start from rest.
``exact`` advances the same inputs with plain torch in 64 bits.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "heatflow-mpm_b200"))

from heatflow_mpm import (AirBatch, AirScenario, AirServer, BoxHeater, GridConfig, Heater, HeatflowMPM,  # noqa: E402
                          Material, Request)
from heatflow_mpm.shapes import Mesh, winding_inside  # noqa: E402

DT = 2e-3
T_AMB = 25.0
EDGES = (32, 48, 64, 96, 128)


def listed():
    sim = dict(kind="sim", L=0.48, heater="trough", radius=0.0, fan=0.0, power=400.0, cg="classic", tol=1e-4, steps=10,
               moving=False)
    return [
        # one substep of a very small coupled box: what a call costs when there is hardly any work in it
        dict(sim, name="box12", n=12, L=0.12, heater="box", radius=0.02, fan=2.0, power=50.0, tol=1e-5, steps=1),
        # the air-only plume at 32^3 with the tight tolerance: latency of many small CG iterations
        dict(sim, name="plume32", n=32, heater="box", tol=1e-6),
        # a coupled scene whose edge is a multiple of nothing
        dict(sim, name="odd75", n=75, radius=0.04, fan=1.0),
        # the default coupled scene: the ten substeps of one output frame
        dict(sim, name="coupled96", n=96, radius=0.04, fan=2.0),
        # the same driven from outside: particle states uploaded and the temperature downloaded every substep
        dict(sim, name="streamed96", n=96, radius=0.04, fan=2.0, cg="single-reduction", moving=True),
        # an air-only room at 128^3
        dict(sim, name="air128", n=128, fan=1.5, power=600.0),
        # the precision-study scene: the largest single scene
        dict(sim, name="coupled160", n=160, radius=0.035, fan=1.0, power=800.0),
        # an ensemble of independent scenes of uneven size, from rest, advanced together
        dict(name="ensemble12", kind="batch", scenes=12, mix=3, steps=20),
        # a few scenes of one small size: a batch that does not fill the device
        dict(name="ensemble4", kind="batch", scenes=4, mix=2, steps=20, edge=48),
        # requests of uneven size and horizon, served until all are done: admission, retirement and results included
        dict(name="served8", kind="serve", requests=8, mix=5, horizon=30),
        # the lattice points of a mesh fill tested against its triangles
        dict(name="fill5k", kind="fill", rings=50, spacing=2.5e-3),
    ]


def draw(rng):
    kind = rng.choice(["sim"] * 6 + ["batch", "batch", "serve", "fill"])
    if kind == "sim":
        n = int(round(math.exp(rng.uniform(math.log(12), math.log(150)))))
        coupled = rng.random() < 0.6
        return dict(kind="sim", n=n, L=0.48, heater="trough" if n >= 40 else "box",
                    radius=round(rng.uniform(0.03, 0.05), 4) if coupled else 0.0, fan=round(rng.uniform(0.0, 3.0), 2),
                    power=round(rng.uniform(100.0, 800.0), 1), cg=rng.choice(["classic", "classic", "single-reduction"]),
                    tol=rng.choice([1e-4, 1e-4, 1e-5]), steps=1 if n <= 32 and rng.random() < 0.4 else rng.choice([4, 10]), moving=coupled and rng.random() < 0.5)
    if kind == "batch":
        c = dict(kind="batch", scenes=rng.randint(2, 10), mix=rng.randint(0, 9999), steps=2 * rng.randint(6, 10))
        if rng.random() < 0.3:
            c["edge"] = rng.choice([40, 50, 72, 80, 100])
        return c
    if kind == "serve":
        return dict(kind="serve", requests=rng.randint(3, 8), mix=rng.randint(0, 9999), horizon=rng.randint(10, 30))
    return dict(kind="fill", rings=rng.randint(12, 60), spacing=round(math.exp(rng.uniform(math.log(2.5e-3), math.log(8e-3))), 5))


# ------------------------------------------------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _heater(case):
    kw = dict(power=case["power"], t_cap=120.0, fan=case["fan"])
    if case["heater"] == "trough":
        return Heater(**kw)
    return BoxHeater(x=0.25 * case["L"], **kw)


def _flow(n, L, rng, speed=0.3):
    """A velocity field on the MAC faces whose discrete divergence is zero and which vanishes on the walls (the curl of
    a random smooth vector potential), and a temperature with a warm plume and fine noise; float32, on the GPU."""
    dev, h = _device(), L / n
    node = torch.arange(n + 1, dtype=torch.float64, device=dev) / n
    mid = (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) / n

    def potential(a, b, c):
        out = torch.zeros((len(a), len(b), len(c)), dtype=torch.float64, device=dev)
        for _ in range(4):
            k, ph, amp = rng.integers(1, 4, 3), rng.uniform(0, 2 * np.pi, 3), rng.normal()
            f = [torch.cos(float(np.pi * kk) * x + float(p)) * torch.sin(math.pi * x) ** 2 for kk, p, x in zip(k, ph, (a, b, c))]
            out += float(amp) * f[0][:, None, None] * f[1][None, :, None] * f[2][None, None, :]
        return out

    px, py, pz = potential(mid, node, node), potential(node, mid, node), potential(node, node, mid)
    u = (pz[:, 1:] - pz[:, :-1]) - (py[:, :, 1:] - py[:, :, :-1])
    v = (px[:, :, 1:] - px[:, :, :-1]) - (pz[1:] - pz[:-1])
    w = (py[1:] - py[:-1]) - (px[:, 1:] - px[:, :-1])
    top = max(float(a.abs().max()) for a in (u, v, w))
    x, y, z = mid[:, None, None], mid[None, :, None], mid[None, None, :]
    cx, cy = (float(c) for c in rng.uniform(0.25, 0.75, 2))
    wide = 0.08 + 0.1 * z
    T = T_AMB + float(rng.uniform(20, 60)) * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / wide ** 2) * torch.exp(-z)
    g = torch.Generator(device=dev).manual_seed(int(rng.integers(1 << 31)))
    T = T + 0.02 * torch.rand(T.shape, generator=g, dtype=torch.float64, device=dev) - 0.01
    return [a.float() for a in (T, *(f * (speed / top) for f in (u, v, w)))]


def _body(radius, L, spacing, rng):
    """A jittered particle lattice in an ellipsoid that stands on the floor at the box centre, and small velocities."""
    semi = radius * np.array([1.0, 0.75, 1.25])
    lo, hi = -semi - spacing, semi + spacing
    ax = [np.arange(lo[d] + spacing / 2, hi[d], spacing) for d in range(3)]
    P = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    P = P[((P / semi) ** 2).sum(1) <= 1.0]
    P = P + rng.uniform(-0.2, 0.2, P.shape) * spacing + [L / 2, L / 2, semi[2] + spacing / 2]
    return P.astype(np.float32), rng.uniform(-0.05, 0.05, P.shape).astype(np.float32)


def _sim_inputs(case, seed):
    """(state, spacing, particle velocities, the body's path): what the substeps of a pass start from."""
    rng = np.random.default_rng([seed, case["n"]])
    flow = _flow(case["n"], case["L"], rng)
    spacing = 2.5e-3 if case["L"] > 0.2 else 5e-3
    pos = vel = np.zeros((0, 3), np.float32)
    if case["radius"]:
        pos, vel = _body(case["radius"], case["L"], spacing, rng)
    # a moving body: every substep's positions drift with the particle velocities
    path = [(pos + np.float32(k * DT) * vel, vel) for k in range(case["steps"])] if case["moving"] else None
    s = _simulation(case, spacing)
    s.set_flow(*flow)
    if len(pos):
        s.set_particles(pos, vel, torch.full((len(pos),), 20.0))
    for _ in range(16):
        s.substep(DT)
    state = dict(T=s.T, u=s.f[0], v=s.f[1], w=s.f[2], p=s.p)
    if len(pos):
        state["ptemp"] = s.ptemp
    return {k: v.float() for k, v in state.items()}, spacing, pos, vel, path


def _simulation(case, spacing):
    n, L = case["n"], case["L"]
    return _Exact(n, L / n, case["tol"], _cells(case["heater"], n, L / n, L, case["fan"], 0.25 * L), case["power"], case["fan"],
                  spacing=spacing)


def _scenarios(case, seed):
    shape, rng = np.random.default_rng(case["mix"]), np.random.default_rng([seed, 7])
    out = []
    for _ in range(case["scenes"] if case["kind"] == "batch" else case["requests"]):
        n = int(shape.choice(EDGES if case["kind"] == "batch" else EDGES[1:]))
        horizon = int(shape.integers(case.get("horizon", 1) // 2, case.get("horizon", 1) + 1))
        kw = dict(power=float(rng.uniform(100, 800)), fan=float(rng.uniform(0.2, 3)), seed=int(rng.integers(1 << 30)))
        if case["kind"] == "batch":
            kw["heater_x"] = float(rng.uniform(0.05, 0.2))
        elif shape.uniform() < 0.5:
            kw["sphere_radius"] = float(rng.uniform(0.02, 0.06))
        out.append(AirScenario(n=case.get("edge", n), horizon=horizon, **kw))
    return out


def _bumpy(rings):
    """A closed bumpy sphere, 10 cm tall, of 2 * rings * (rings - 1) triangles or so, standing at z = 0."""
    k, ph, amp = (2, 3, 5, 4), (0.3, 1.1, 2.9, 4.4), (0.05, 0.03, 0.02, 0.04)
    th, fi = np.pi * np.arange(1, rings) / rings, 2 * np.pi * np.arange(rings) / rings
    t, f = np.meshgrid(th, fi, indexing="ij")
    r = 1.0 + sum(a * np.sin(kk * f + p) * np.sin(t) ** 2 for kk, p, a in zip(k, ph, amp))
    V = np.stack([r * np.sin(t) * np.cos(f), r * np.sin(t) * np.sin(f), r * np.cos(t)], -1).reshape(-1, 3)
    V = np.concatenate([V, [[0, 0, 1.0], [0, 0, -1.0]]])
    i, j = np.meshgrid(np.arange(rings - 2), np.arange(rings), indexing="ij")
    a, b = i * rings + j, i * rings + (j + 1) % rings
    c, d = a + rings, b + rings
    top, last = len(V) - 2, (rings - 2) * rings
    j = np.arange(rings)
    F = np.concatenate([np.stack([a, c, b], -1).reshape(-1, 3), np.stack([b, c, d], -1).reshape(-1, 3),
                        np.stack([np.full(rings, top), j, (j + 1) % rings], -1),
                        np.stack([np.full(rings, top + 1), last + (j + 1) % rings, last + j], -1)])
    V = V * 0.05
    V[:, 2] -= V[:, 2].min()
    return V, F.astype(np.int64)


def _fill_points(case, seed):
    """The mesh and the jittered lattice over its bounds that a fill tests."""
    V, F = _bumpy(case["rings"])
    sp = case["spacing"]
    lo, hi = V.min(0) - sp, V.max(0) + sp
    ax = [np.arange(lo[d] + sp / 2, hi[d], sp) for d in range(3)]
    P = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    return V, F, (P + np.random.default_rng(seed).uniform(-0.2, 0.2, P.shape) * sp).astype(np.float32)


# ------------------------------------------------------------------------------------------------------------ passes
def prepare(case, seed):
    if case["kind"] == "fill":
        V, F, points = _fill_points(case, seed)
        return dict(case=case, mesh=Mesh(V, F), points=points)
    if case["kind"] == "batch":
        batch = AirBatch(_scenarios(case, seed))
        return dict(case=case, batch=batch, saved=batch.snapshot(), par=[sc.parity() for sc in batch.scenes])
    if case["kind"] == "serve":
        return dict(case=case, scenarios=_scenarios(case, seed))
    saved, spacing, pos, vel, path = _sim_inputs(case, seed)
    sim = HeatflowMPM(pos, mat=Material(t_sol=28.0, t_liq=34.0), heater=_heater(case),
                      grid=GridConfig(L=case["L"], h=case["L"] / case["n"], cg_tol=case["tol"]), spacing=spacing, body="frozen",
                      particle_velocities=vel, cg=case["cg"])
    _load(sim.scene, saved, sim.scene.parity())
    state = dict(case=case, sim=sim, saved=saved, par=sim.scene.parity())
    if path is not None:
        state["path"] = [tuple(torch.from_numpy(a).pin_memory() for a in step) for step in path]
        state["down"] = [torch.empty((case["n"],) * 3).pin_memory() for _ in path]
    return state


def _load(scene, saved, par):
    """Put a saved state into the current buffers of a scene."""
    for name in ("T", "u", "v", "w"):
        getattr(scene, name)[par].copy_(saved[name])
    scene.p.copy_(saved["p"])
    if "ptemp" in saved:
        scene.ptemp.copy_(saved["ptemp"])


def _current(scene, par):
    return dict(T=scene.T[par], u=scene.u[par], v=scene.v[par], w=scene.w[par], p=scene.p)


def run(state):
    case = state["case"]
    if case["kind"] == "fill":
        return winding_inside(state["mesh"], state["points"], return_winding=True)
    if case["kind"] == "batch":
        batch = state["batch"]
        for sc, saved, par in zip(batch.scenes, state["saved"], state["par"]):
            _load(sc, saved, par)
        batch.run(DT, case["steps"])
        state["par"] = [sc.parity() for sc in batch.scenes]
        return [_current(sc, par) for sc, par in zip(batch.scenes, state["par"])]
    if case["kind"] == "serve":
        server = AirServer(dt=DT, max_slots=64, keep_results=True)
        trace = [Request(sc, 0.0, rid=i) for i, sc in enumerate(state["scenarios"])]
        server.serve(trace)
        return [{k: r.result[k] for k in ("T", "u", "v", "w")} for r in trace]
    sim = state["sim"]
    if case["steps"] > 1:
        _load(sim.scene, state["saved"], state["par"])
    if "path" in state:
        for (pos, vel), down in zip(state["path"], state["down"]):
            sim.body.set_state(pos, vel)
            sim.substep(DT)
            landed = sim.grid_T_async(down)
        landed.synchronize()
    else:
        for _ in range(case["steps"]):
            sim.substep(DT)
    state["par"] = sim.scene.parity()
    out = _current(sim.scene, state["par"])
    if sim.n:
        out["ptemp"], out["pmelt"] = sim.scene.ptemp, sim.scene.pmelt
    if "path" in state:
        out["host_T"] = state["down"]
    return out


def work(case):
    """Bytes: each field of the state (T, u, v, w, p) read and written once per substep, the obstacle fields, fixed cells
    and their values read once, particles read and written once.  Flops: about 28 trilinear samples per cell, and the CG
    iterations, whose number grows like the edge (about n / 2 at the usual tolerance)."""
    if case["kind"] == "fill":
        tri = 2 * case["rings"] * (case["rings"] - 1)
        points = 0.12 ** 3 / case["spacing"] ** 3
        return dict(bytes=36.0 * tri + 16.0 * points, flops=60.0 * tri * points)
    if case["kind"] == "sim":
        scenes = [(case["n"], case["steps"], case["radius"] ** 3 * 4 / 1.5625e-8 if case["radius"] else 0.0, case["tol"])]
    else:
        scenes = [(s.n, case.get("steps", s.horizon), 0.0, 1e-4) for s in _scenarios(case, 0)]
    total = dict(bytes=0.0, flops=0.0)
    for n, steps, particles, tol in scenes:
        its = 0.5 * n * math.log10(tol) / -4
        total["bytes"] += steps * (4.0 * n ** 3 * 18.25 + 4.0 * particles * 12)
        total["flops"] += steps * (n ** 3 * (28 * 45 + 30.0 * its) + particles * 700)
    return total


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    if case["kind"] == "fill":
        return _exact_fill(case, seed)
    if case["kind"] == "sim":
        saved, spacing, pos, vel, path = _sim_inputs(case, seed)
        s = _simulation(case, spacing)
        s.set_flow(*(saved[k] for k in "Tuvwp"))
        if len(pos):
            s.set_particles(pos, vel, saved["ptemp"])
        shown = []
        for k in range(case["steps"]):
            if path is not None:
                s.move(*path[k])
            s.substep(DT)
            shown.append(s.T.cpu())
        out = dict(T=s.T, u=s.f[0], v=s.f[1], w=s.f[2], p=s.p)
        if len(pos):
            out["ptemp"], out["pmelt"] = s.ptemp, s.pmelt
        if path is not None:
            out["host_T"] = shown
        return out
    outs = []
    for sc in _scenarios(case, seed):
        kind = "trough" if sc.heater_x is None else "box"
        s = _Exact(sc.n, 0.48 / sc.n, 1e-4, _cells(kind, sc.n, 0.48 / sc.n, 0.48, sc.fan, sc.heater_x), sc.power, sc.fan,
                   ball=sc.sphere_radius)
        noise = np.random.default_rng(sc.seed).uniform(-0.01, 0.01, (sc.n,) * 3)
        s.set_flow((T_AMB + noise).astype(np.float32))
        for _ in range(case.get("steps", sc.horizon)):
            s.substep(DT)
        out = dict(T=s.T, u=s.f[0], v=s.f[1], w=s.f[2])
        if case["kind"] == "batch":
            out["p"] = s.p
        outs.append({k: v.cpu() for k, v in out.items()})
    return outs


def _cells(kind, n, h, L, fan, x):
    """Cell classes 0 air, 1 shell, 2 rod, 3 fan outlet, 4 trough air, and the direction that the heater faces."""
    c = np.zeros((n, n, n), np.int32)
    if kind == "box":
        i, j = int(round(x / h)) - 2, int(round(L / 2 / h)) - 2
        c[i:i + 4, j:j + 4, :2], c[i:i + 4, j:j + 4, 2] = 2, 4
        if fan > 0:
            c[i:i + 4, j:j + 4, 3] = 3
        return c, np.array([0.0, 0.0, 1.0])
    R, half, tilt = 0.055, 0.11, math.radians(15.0)
    d = np.array([-0.423, 0.906]) / np.linalg.norm([-0.423, 0.906])
    centre = np.array([L / 2 + 0.21 * d[0], L / 2 + 0.21 * d[1], 0.12])
    facing = np.array([-d[0] * np.cos(tilt), -d[1] * np.cos(tilt), -np.sin(tilt)])
    axis = np.array([d[1], -d[0], 0.0])
    g = (np.arange(n) + 0.5) * h
    rel = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1) - centre
    s, q, r = rel @ axis, rel @ facing, rel @ np.cross(axis, facing)
    rad = np.hypot(q, r)
    c[(abs(s) <= half) & (q <= 0) & (rad >= R - h / 2) & (rad <= R + 0.006 + h / 2)] = 1
    c[(abs(abs(s) - half) <= h / 2) & (q <= 0) & (rad <= R + 0.006)] = 1
    for z in (-0.03, 0.03):
        c[(abs(s) <= half - 0.015) & (np.hypot(q + 0.03, r - z) <= 0.007 + h / 2)] = 2
    if fan > 0:
        c[(c == 0) & (abs(s) <= half - 0.02) & (abs(r) <= R - 0.01) & (q > 0) & (q <= 0.015)] = 3
    c[(c == 0) & (abs(s) <= half - 0.015) & (rad <= R - 0.004) & (q <= 0)] = 4
    return c, facing


class _Exact:
    """The air substep in 64 bits: temperature rebuild, heat source, semi-Lagrangian advection, implicit diffusion,
    particle temperatures, buoyancy, relaxation toward the obstacles and the pressure projection, both linear systems
    by Jacobi-preconditioned CG to their relative tolerances."""

    def __init__(self, n, h, tol, cells, power, fan, spacing=2.5e-3, ball=0.0):
        self.n, self.h, self.tol, self.dev = n, h, tol, _device()
        cell, facing = cells
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)
        wall = np.zeros((n, n, n), bool)
        wall[[0, -1]] = wall[:, [0, -1]] = True
        wall[:, :, -1] = True
        solid, source, rod = (cell == 1) | (cell == 2), cell >= 3, cell == 2
        fixed, tfix = rod | wall, np.where(rod, 300.0, np.where(wall, T_AMB, 0.0))
        g = (np.arange(n) + 0.5) * h
        c = 0.5 * n * h
        inside = (np.zeros((n, n, n), bool) if not ball else
                  (g[:, None, None] - c) ** 2 + (g[None, :, None] - c) ** 2 + (g[None, None, :] - ball) ** 2 <= ball * ball)
        self.st_k, self.st_m = [], []
        for a in range(3):
            touch = lambda m: np.concatenate([m, np.zeros_like(np.take(m, [0], a))], a) | \
                np.concatenate([np.zeros_like(np.take(m, [0], a)), m], a)
            on, blown, on_ball = touch(solid), touch(cell == 3), touch(inside)
            blown &= ~on
            k, m = np.where(on, 1.0, np.where(blown, 0.05, 0.0)), np.where(blown, 0.05 * fan * facing[a], 0.0)
            self.st_k.append(t(np.where(on_ball, 1.0, k)))
            self.st_m.append(t(np.where(on_ball, 0.0, m)))
        self.st_alpha = t((solid | inside).astype(np.float64))
        self.fixed, self.tfix, self.source = t(fixed | inside), t(np.where(inside, 20.0, tfix)), t(source)
        self.rate = power / (1.2 * 1005.0 * max(int(source.sum()), 1) * h ** 3)
        self.vol, self.pos = spacing ** 3, None
        zero = lambda *s: torch.zeros(s, dtype=torch.float64, device=self.dev)
        self.shapes = [(n + 1, n, n), (n, n + 1, n), (n, n, n + 1)]
        self.f, self.p = [zero(*s) for s in self.shapes], zero(n, n, n)
        g = torch.arange(n + 1, dtype=torch.float64, device=self.dev) * h
        self.node, self.mid = g, (g + 0.5 * h)[:n]

    def set_flow(self, T, u=None, v=None, w=None, p=None):
        d = lambda a: torch.as_tensor(a, device=self.dev).double()
        self.T = torch.where(self.fixed, self.tfix, d(T))
        if u is not None:
            self.f = [d(a) for a in (u, v, w)]
        if p is not None:
            self.p = d(p)

    def set_particles(self, pos, vel, temp):
        self.move(pos, vel)
        self.ptemp = temp.to(self.dev).double()

    def move(self, pos, vel):
        self.pos, self.vel = (torch.as_tensor(a, device=self.dev).double() for a in (pos, vel))

    OFF = ((0.0, 0.5, 0.5), (0.5, 0.0, 0.5), (0.5, 0.5, 0.0), (0.5, 0.5, 0.5))

    def _corners(self, x, off, shape):
        """The eight lattice nodes around each point, clamped to the lattice, and their trilinear weights."""
        lo, hi = [], []
        for d in range(3):
            g = x[d] / self.h - off[d]
            i = torch.floor(g)
            w, i = g - i, i.long()
            lo.append((i.clamp(0, shape[d] - 1), 1.0 - w))
            hi.append(((i + 1).clamp(0, shape[d] - 1), w))
        for a in (lo[0], hi[0]):
            for b in (lo[1], hi[1]):
                for c in (lo[2], hi[2]):
                    yield (a[0] * shape[1] + b[0]) * shape[2] + c[0], a[1] * b[1] * c[1]

    def _sample(self, field, x, off):
        flat, out = field.reshape(-1), 0.0
        for at, w in self._corners(x, off, field.shape):
            out = out + w * flat[at]
        return out

    def _scatter(self, value, off, shape):
        at, w = (torch.stack(a).reshape(-1).cpu().numpy() for a in zip(*self._corners(self.pos.T, off, shape)))
        out = np.bincount(at, w * np.tile(value.cpu().numpy(), 8), math.prod(shape))   # the same order every time
        return torch.as_tensor(out, device=self.dev).reshape(shape)

    def _back(self, x, dt):
        """Where the point x came from: the midpoint rule through the current velocity field."""
        speed = lambda y: [self._sample(self.f[d], y, self.OFF[d]) for d in range(3)]
        half = [a - 0.5 * dt * b for a, b in zip(x, speed(x))]
        return [a - dt * b for a, b in zip(x, speed(half))]

    @staticmethod
    def _low(a, d):
        return a.narrow(d, 0, a.shape[d] - 1)

    @staticmethod
    def _high(a, d):
        return a.narrow(d, 1, a.shape[d] - 1)

    def _faces(self, inner):
        """Three face arrays with the given interior values and zero walls."""
        out = []
        for d, a in enumerate(inner):
            f = torch.zeros(self.shapes[d], dtype=torch.float64, device=self.dev)
            f.narrow(d, 1, self.n - 1).copy_(a)
            out.append(f)
        return out

    def _jumps(self, x):
        return [self._high(x, d) - self._low(x, d) for d in range(3)]

    def _spread(self, inner):
        """Sum over a cell's faces of an interior-face quantity, low faces taken with a plus and high ones with a minus."""
        out = torch.zeros((self.n,) * 3, dtype=torch.float64, device=self.dev)
        for d, a in enumerate(inner):
            out.narrow(d, 1, self.n - 1).add_(a)
            out.narrow(d, 0, self.n - 1).sub_(a)
        return out

    def _total(self, inner):
        out = torch.zeros((self.n,) * 3, dtype=torch.float64, device=self.dev)
        for d, a in enumerate(inner):
            out.narrow(d, 1, self.n - 1).add_(a)
            out.narrow(d, 0, self.n - 1).add_(a)
        return out

    @staticmethod
    def _cg(apply, b, x, D, tol, most):
        r, x = b - apply(x), x.clone()
        z = D * r
        p, rz, rr = z.clone(), float((r * z).sum()), float((r * r).sum())
        stop = max(tol * math.sqrt(float((b * b).sum())), tol, 1e-18) ** 2
        for _ in range(most + (most & 1)):
            if not rr > stop:
                break
            Ap = apply(p)
            a = rz / float((p * Ap).sum())
            x.add_(p, alpha=a)
            r.add_(Ap, alpha=-a)
            z = D * r
            rr, new = torch.stack(((r * r).sum(), (r * z).sum())).tolist()
            p.mul_(new / rz).add_(z)
            rz = new
        return x

    def substep(self, dt):
        n, h, fixed = self.n, self.h, self.fixed
        alpha_s, k, m, q = self.st_alpha, self.st_k, self.st_m, [torch.zeros(s, dtype=torch.float64, device=self.dev) for s in self.shapes]
        Tw = self.T
        if self.pos is not None:
            one = torch.ones(len(self.pos), dtype=torch.float64, device=self.dev)
            part = self.vol / h ** 3
            alpha = self._scatter(part * one, self.OFF[3], (n, n, n))
            alpha_s = alpha_s + alpha
            k = [a + self._scatter(1e-3 * one, self.OFF[d], self.shapes[d]) for d, a in enumerate(k)]
            m = [a + self._scatter(1e-3 * self.vel[:, d], self.OFF[d], self.shapes[d]) for d, a in enumerate(m)]
            q = [self._scatter(part * self.vel[:, d], self.OFF[d], self.shapes[d]) for d in range(3)]
            q = self._faces([q[d].narrow(d, 1, n - 1) for d in range(3)])
            warm = self._scatter(part * self.ptemp, self.OFF[3], (n, n, n))
            Tw = torch.where(alpha > 0.05, warm / alpha.clamp(min=1e-30), Tw)
        open_ = [(1.0 - 0.5 * (self._low(alpha_s, d) + self._high(alpha_s, d))).clamp(0.05, 1.0) for d in range(3)]
        kap = 2.2e-5 + (2.0e-5 - 2.2e-5) * (alpha_s / 0.6).clamp(0.0, 1.0)
        hk = [2 * self._low(kap, d) * self._high(kap, d) / (self._low(kap, d) + self._high(kap, d) + 1e-12) for d in range(3)]
        # temperature: fixed cells, heat source, advection, diffusion
        Tw = torch.where(fixed, self.tfix, Tw)
        if self.rate > 0:
            Tw = torch.where(self.source, torch.minimum(Tw + self.rate * dt, Tw.clamp(min=120.0)), Tw)
        grid = lambda a, b, c: torch.meshgrid(a, b, c, indexing="ij")
        moved = self._sample(Tw, self._back(grid(self.mid, self.mid, self.mid), dt), self.OFF[3])
        T = torch.where(alpha_s > 0.5, Tw, moved)
        c, free = dt / h ** 2, ~fixed
        known = torch.where(fixed, self.tfix, torch.zeros_like(T))
        both = [self._low(free, d) & self._high(free, d) for d in range(3)]
        kfree = [torch.where(b, a, torch.zeros_like(a)) for a, b in zip(hk, both)]
        ktouch = self._total([torch.where(b, torch.zeros_like(a), a) for a, b in zip(hk, both)])
        near = torch.zeros_like(T)
        for d in range(3):
            near.narrow(d, 1, n - 1).add_(hk[d] * self._low(known, d))
            near.narrow(d, 0, n - 1).add_(hk[d] * self._high(known, d))
        b = torch.where(fixed, self.tfix, T + c * near)
        apply = lambda x: torch.where(fixed, x, x + c * (self._spread([a * j for a, j in zip(kfree, self._jumps(x))]) + ktouch * x))
        D = torch.where(fixed, torch.ones_like(T), 1.0 / (1.0 + c * self._total(hk)))
        T = self._cg(apply, b, T, D, 1e-6, 200)
        if self.pos is not None:
            x = self.pos.T
            change = self._sample(T, x, self.OFF[3]) - self._sample(Tw, x, self.OFF[3])
            self.ptemp = (self.ptemp + change).clamp(0.0, 300.0)
            self.pmelt = ((self.ptemp - 28.0) / 6.0).clamp(0.0, 1.0)
        # faces: advection, buoyancy, relaxation
        new = []
        for d in range(3):
            at = [self.mid] * 3
            at[d] = self.node[1:n]
            val = self._sample(self.f[d], self._back(grid(*at), dt), self.OFF[d])
            if d == 2:
                val = val + dt * 9.81 * (0.5 * (self._low(T, 2) + self._high(T, 2)) - T_AMB) / (T_AMB + 273.15)
            s = dt / (1.2 * open_[d] * h ** 3)
            new.append((val + s * m[d].narrow(d, 1, n - 1)) / (1.0 + s * k[d].narrow(d, 1, n - 1)))
        # pressure projection
        flux = [a * f + g.narrow(d, 1, n - 1) for d, (a, f, g) in enumerate(zip(open_, new, q))]
        rhs = (1.2 / dt) * self._spread(flux) / h
        rhs = rhs - rhs.mean()
        lap = lambda x: self._spread([a * j for a, j in zip(open_, self._jumps(x))]) / h ** 2
        self.p = self._cg(lap, rhs, self.p, h ** 2 / self._total(open_).clamp(min=1e-12), self.tol, 400)
        self.f = self._faces([f - dt / 1.2 * j / h for f, j in zip(new, self._jumps(self.p))])
        self.T = T


def _exact_fill(case, seed):
    V, F, P = _fill_points(case, seed)
    dev = _device()
    tri, total = torch.as_tensor(V[F], device=dev), torch.zeros(len(P), dtype=torch.float64, device=dev)
    pts = torch.as_tensor(P, device=dev).double()
    for t in tri.split(128):
        a, b, c = (t[None, :, i] - pts[:, None] for i in range(3))
        la, lb, lc = (x.norm(dim=-1) for x in (a, b, c))
        num = (a * torch.linalg.cross(b, c)).sum(-1)
        den = la * lb * lc + (a * b).sum(-1) * lc + (b * c).sum(-1) * la + (c * a).sum(-1) * lb
        total += torch.atan2(num, den).sum(1) / (2 * math.pi)
    return (total > 0.5).cpu().numpy(), total.cpu().numpy()
