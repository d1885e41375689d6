"""The work that programs have this library do, as cases whose time and outputs can be measured.

listed() gives the cases, draw(rng) more of the same ranges, prepare(case, seed) what a program has in hand
before the call (its solver and inputs, made from the seed), run(state) one pass through the public entry
points with the outputs whole, work(case) the bytes and operations a pass cannot do without, and
exact(case, seed) the outputs in 64-bit arithmetic, from a restatement of the substep in plain torch.

Kinds of case:
  tank       the SI water tank (Tait water, no-slip walls): substeps, then the particles read back
  dam        the two-phase water/oil dam break (linear EOS), default or fixed-point transfer
  materials  one block of each of the six constitutive models
  gate4      the multi-material scene with pebbles (bonded triangles) and fracture bonds
  tanks      many tanks of uneven size in one batched solver
  surface    a macrostep of the dam break, then the free-surface field a renderer draws
  adjoint    one step of a fit: initial velocities in, trajectory loss and its gradients out
`restart` cases put the particles back to their start before stepping (episodes, parameter studies); the
others go on from where the last pass ended, as a simulation that saves its state every so often does.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "powder-play_b200"))

from mpm_b200 import (calculate_mpm_cfl_microsteps, create_experimental_mpm_mls_atomic_gpu_solver,  # noqa: E402
                      create_mpm_batched_gpu_solver, create_mpm_mls_gpu_solver)
from mpm_b200.adjoint import create_mpm_adjoint_engine  # noqa: E402
from mpm_b200.layout import ParticleArrays  # noqa: E402
from mpm_b200.scenes import create_mpm_gate4_scene, create_mpm_gate4_step_config  # noqa: E402

# SI tank water: 1000 kg/m^3 and 20 m/s over 0.02 m of depth, gamma 7
TAIT = {"lambda": 1000.0 * 400.0 / 7.0 * 0.02, "mu": 0.0, "model": "water", "density": 20.0,
        "equationOfState": {"model": "tait", "exponent": 7.0}}
WATER = {"lambda": 160_000.0, "mu": 0.0, "model": "water", "density": 0.02}
OIL = {"lambda": 120_000.0, "mu": 0.0, "model": "oil", "density": 0.016}
ADJOINT_WATER = {"lambda": 22_857.0, "mu": 0.0, "model": "water", "density": 0.02,
                 "equationOfState": {"model": "tait", "exponent": 7.0}}
ADJOINT_SOLID = {"lambda": 20.0, "mu": 10.0, "model": "fixed-corotated"}
SIX = [{"lambda": 20.0, "mu": 10.0, "model": "neo-hookean"},
       {"lambda": 20.0, "mu": 10.0, "model": "snow"},
       {"lambda": 8.0, "mu": 0.0, "model": "water", "density": 1.0},
       {"lambda": 6.0, "mu": 0.0, "model": "oil", "density": 0.8},
       {"lambda": 20.0, "mu": 10.0, "model": "powder", "frictionCoefficient": 0.55},
       {"lambda": 20.0, "mu": 10.0, "model": "fixed-corotated"}]
TANK_GRAVITY = {"x": 0.0, "y": -9.81}
DAM_GRAVITY = {"x": 0.0, "y": 90.0}
NO_LIMIT = 1 << 20  # microsteps a plan may take


def listed():
    return [
        # the smallest call: a few substeps of the 1,600-particle tank, between two looks at its state
        {"name": "tank_4", "kind": "tank", "particles": 1600, "side": 80, "steps": 4, "restart": False},
        # the same tank over a whole macrostep of 1/120 s under its CFL guard: launch after launch
        {"name": "tank_macrostep", "kind": "tank", "particles": 1600, "side": 80, "steps": 0, "restart": False},
        # an episode of a larger tank on an odd grid, started over each time
        {"name": "tank_episode", "kind": "tank", "particles": 20011, "side": 197, "steps": 32, "restart": True},
        # a dam break of ordinary size, ragged in particles and grid, started over each time
        {"name": "dam_150k", "kind": "dam", "particles": 150_002, "columns": 211, "steps": 40, "restart": True,
         "fixed": False},
        # the million-particle dam break, a saved state every 200 substeps
        {"name": "dam_1m", "kind": "dam", "particles": 1_000_000, "columns": 500, "steps": 200, "restart": False,
         "fixed": False},
        # the order-independent integer transfer
        {"name": "dam_fixed", "kind": "dam", "particles": 240_000, "columns": 300, "steps": 40, "restart": True,
         "fixed": True},
        # every constitutive model at once
        {"name": "materials", "kind": "materials", "particles": 48_006, "steps": 24},
        # the interactive scene: two liquids, 50 pebbles, a breakable block; one macrostep of 5 substeps
        {"name": "gate4", "kind": "gate4", "diameter": 20.0, "steps": 5},
        # many small simulations advanced together, each read back
        {"name": "tanks_24", "kind": "tanks", "scenes": 24, "particles": 16_000, "steps": 48},
        # a rendered frame: a macrostep of 1/240 s, then the water and oil area of every node
        {"name": "surface_frame", "kind": "surface", "particles": 240_000, "columns": 300},
        # a fit of one small scene, the whole trajectory kept
        {"name": "fit_1k", "kind": "adjoint", "scenes": 1, "columns": 24, "rows": 32, "solid": 16, "cells": 64,
         "steps": 40, "every": 40},
        # a fit over 64 scenes of 16,384 particles with a checkpoint every 20 of 200 substeps
        {"name": "fit_64", "kind": "adjoint", "scenes": 64, "columns": 96, "rows": 128, "solid": 64, "cells": 256,
         "steps": 200, "every": 20},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["tank", "tank", "dam", "dam", "dam", "fixed", "materials", "gate4", "tanks", "surface",
                       "adjoint", "adjoint"])
    if kind == "tank":
        return {"kind": "tank", "particles": log(1000, 64_000), "side": rng.randint(64, 512), "steps": log(1, 300),
                "restart": rng.random() < 0.5}
    if kind in ("dam", "fixed"):
        n = log(4000, 240_000 if kind == "fixed" else 1_000_000)
        columns = max(20, int(math.sqrt(n) * rng.uniform(0.3, 0.8)))
        steps = max(1, min(log(4, 300), 200_000_000 // n))
        return {"kind": "dam", "particles": n, "columns": columns, "steps": steps, "restart": True,
                "fixed": kind == "fixed"}
    if kind == "materials":
        return {"kind": "materials", "particles": log(600, 60_000), "steps": log(4, 60)}
    if kind == "gate4":
        return {"kind": "gate4", "diameter": round(rng.uniform(10.0, 21.0), 2), "steps": rng.randint(1, 8)}
    if kind == "tanks":
        return {"kind": "tanks", "scenes": rng.randint(2, 24), "particles": log(2000, 16_000), "steps": log(8, 100)}
    if kind == "surface":
        n = log(4000, 400_000)
        return {"kind": "surface", "particles": n, "columns": max(20, int(math.sqrt(n) * rng.uniform(0.3, 0.8)))}
    scenes = log(1, 48)
    steps = log(10, 200)
    return {"kind": "adjoint", "scenes": scenes, "columns": rng.randint(16, 96), "rows": rng.randint(16, 128),
            "solid": rng.randint(8, 64), "cells": 256, "steps": steps,
            "every": steps if rng.random() < 0.3 else rng.randint(5, 25)}


# ------------------------------------------------------------------ scenes --

def f32(v):
    return float(np.float32(v))


def blank(n, volume):
    p = ParticleArrays.empty(n)
    p.volume[:] = volume
    p.plastic_volume[:] = 1.0
    return p


def tank(n, side, rng):
    """n particles of Tait water at about 2 x 2 per cell in a 0.2 m box of side x side cells: a jittered
    block in the lower left, with a slow swirl."""
    dx = 0.2 / side
    width = 0.11
    spacing = min(dx / 2, math.sqrt(width * 0.12 / n))
    columns = min(n, max(1, int(width / spacing)))
    r, c = np.divmod(np.arange(n), columns)
    p = blank(n, spacing * spacing)
    p.px[:] = (c + 0.5 + rng.uniform(-0.2, 0.2, n)) * spacing
    p.py[:] = (r + 0.5 + rng.uniform(-0.2, 0.2, n)) * spacing
    k, a = 2 * math.pi / 0.1, rng.uniform(0, 2 * math.pi, 2)
    p.vx[:] = 0.2 * np.sin(k * p.py + a[0])
    p.vy[:] = 0.2 * np.sin(k * p.px + a[1])
    config = {"grid": {"cellsX": side, "cellsY": side, "cellSize": dx}, "particleMass": TAIT["density"] * spacing ** 2,
              "particleVolume": spacing * spacing, "material": TAIT, "wallFriction": 1.0}
    return p, config


def dam(n, columns, rng):
    """n particles, the lower half water and the upper half oil, at 2 x 2 per cell of 10 against the left
    wall; the grid leaves as much room again on the right and above (the 1,000,000-particle scene: 500
    columns on 1024 x 2048 cells)."""
    spacing, dx = 5.0, 10.0
    half = n // 2
    rows = -(-half // columns), -(-(n - half) // columns)
    big = n == 1_000_000 and columns == 500
    cells_x = 1024 if big else columns + columns // 7 + 9
    cells_y = 2048 if big else (rows[0] + rows[1]) * 5 // 7 + 11
    height = cells_y * dx
    r, c = np.divmod(np.concatenate([np.arange(half), np.arange(n - half)]), columns)
    r[half:] += rows[0]
    p = blank(n, spacing * spacing)
    p.px[:] = 20.0 + (c + 0.5 + rng.uniform(-0.2, 0.2, n)) * spacing
    p.py[:] = height - 20.0 - (r + 0.5 + rng.uniform(-0.2, 0.2, n)) * spacing
    k, a = 2 * math.pi / (columns * spacing), rng.uniform(0, 2 * math.pi, 2)
    p.vx[:] = 40.0 * np.sin(k * p.py + a[0])
    p.vy[:] = 40.0 * np.sin(k * p.px + a[1])
    p.materials = [WATER, OIL]
    p.material[:half], p.material[half:] = 0, 1
    p.object_id[:half], p.object_id[half:] = 1, 2
    config = {"grid": {"cellsX": cells_x, "cellsY": cells_y, "cellSize": dx}, "particleMass": WATER["density"] * 25.0,
              "particleVolume": 25.0, "material": WATER, "wallFriction": 0.0}
    return p, config


def materials(n, rng):
    """A block of each model on cells of 1 at 2 x 2 per cell, slightly deformed and moving; the water and
    the oil are near enough to share nodes."""
    each = n // 6
    columns = max(2, int(math.sqrt(each)))
    rows = -(-each // columns)
    p = blank(6 * each, 0.25)
    p.materials = [dict(m) for m in SIX]
    k = np.arange(each)
    r, c = np.divmod(k, columns)
    wide = columns * 0.5 + 3.0
    for m in range(6):
        s = slice(m * each, (m + 1) * each)
        x0 = 4.0 + m * wide - (2.6 if m == 3 else 0.0)
        p.px[s] = x0 + (c + 0.5 + rng.uniform(-0.1, 0.1, each)) * 0.5
        p.py[s] = 4.0 + (r + 0.5 + rng.uniform(-0.1, 0.1, each)) * 0.5
        a = rng.uniform(0, 2 * math.pi, 2)
        p.vx[s] = 0.4 * np.sin(0.3 * p.py[s] + a[0])
        p.vy[s] = 0.4 * np.sin(0.3 * p.px[s] + a[1])
        p.material[s] = m
        p.object_id[s] = m + 1
    p.F[:] += rng.uniform(-0.03, 0.03, p.F.shape)
    config = {"grid": {"cellsX": int(6 * wide) + 8, "cellsY": int(rows * 0.5) + 13, "cellSize": 1.0},
              "particleMass": 0.25, "particleVolume": 0.25, "material": SIX[0], "wallFriction": 0.3}
    return p, config


def fit_scene(case, rng):
    """A water and a solid block at 2 x 2 per cell of 10 in the two halves of the grid."""
    size, spacing = case["cells"] * 10.0, 5.0
    w, h, s = case["columns"], case["rows"], case["solid"]

    def place(lo, extent, room):
        return lo + 40.0 + rng.uniform(0, 1) * max(0.0, room - extent - 80.0)

    p = blank(w * h + s * s, spacing * spacing)
    r, c = np.divmod(np.arange(w * h), w)
    p.px[:w * h] = place(0.0, w * spacing, size / 2) + (c + 0.5) * spacing
    p.py[:w * h] = place(0.0, h * spacing, size) + (r + 0.5) * spacing
    r, c = np.divmod(np.arange(s * s), s)
    p.px[w * h:] = place(size / 2, s * spacing, size / 2) + (c + 0.5) * spacing
    p.py[w * h:] = place(0.0, s * spacing, size) + (r + 0.5) * spacing
    p.vx[:], p.vy[:] = rng.normal(0, 10, len(p)), rng.normal(0, 10, len(p))
    p.materials = [ADJOINT_WATER, ADJOINT_SOLID]
    p.material[:w * h], p.material[w * h:] = 0, 1
    p.object_id[:w * h], p.object_id[w * h:] = 1, 2
    a = rng.uniform(0, 2 * math.pi, 2)
    targets = np.stack([p.px + 20 * np.sin(2 * math.pi * p.px / size + a[0]),
                        p.py + 20 * np.cos(2 * math.pi * p.py / size + a[1])], axis=1).astype(np.float32)
    config = {"grid": {"cellsX": case["cells"], "cellsY": case["cells"], "cellSize": 10.0}, "particleMass": 0.5,
              "particleVolume": 25.0, "material": ADJOINT_SOLID, "wallFriction": 0.0}
    return p, config, targets


FIT_DT = 0.3 * 10.0 / (2828.0 + 60.0)
TANK_BOUNDS = {"waveSpeedBound": 30.0, "velocityBound": 3.0}  # room above the rest values of 20 and about 0.3 m/s
DAM_WAVE, DAM_SPEED = 2840.0, 1500.0


def scene_of(case, seed):
    """(particles, config, dt, gravity) of the single-scene kinds."""
    rng = np.random.default_rng([seed, 17])
    kind = case["kind"]
    if kind == "tank":
        p, config = tank(case["particles"], case["side"], rng)
        return p, config, 0.3 * config["grid"]["cellSize"] / 33.0, TANK_GRAVITY
    if kind in ("dam", "surface"):
        p, config = dam(case["particles"], case["columns"], rng)
        return p, config, 0.3 * 10.0 / (DAM_WAVE + DAM_SPEED), DAM_GRAVITY
    if kind == "materials":
        p, config = materials(case["particles"], rng)
        return p, config, 0.01, {"x": 0.0, "y": -1.0}
    raise ValueError(kind)


def tank_scenes(case, seed):
    """Scene k of a batch: particles log-uniform between 1,000 and the case's most and grid side 64 to 320, by
    k alone; the particles themselves by the seed."""
    out = []
    for k in range(case["scenes"]):
        size = np.random.default_rng([29, k])
        n = int(round(math.exp(size.uniform(math.log(1000), math.log(case["particles"])))))
        out.append(tank(n, int(size.integers(64, 321)), np.random.default_rng([seed, 29, k])))
    return out


# ----------------------------------------------------------- prepare and run --

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "tanks":
        scenes = tank_scenes(case, seed)
        s["solver"] = create_mpm_batched_gpu_solver(scenes)
        s["steps"] = [case["steps"]] * len(scenes)
        s["dts"] = [0.3 * c["grid"]["cellSize"] / 33.0 for _, c in scenes]
        return s
    if kind == "adjoint":
        scenes = [fit_scene(case, np.random.default_rng([seed, 31, k])) for k in range(case["scenes"])]
        s["engine"] = create_mpm_adjoint_engine([(p, c) for p, c, _ in scenes], DAM_GRAVITY)
        s["velocities"] = np.concatenate([np.stack([p.vx, p.vy], axis=1) for p, _, _ in scenes]).astype(np.float32)
        s["targets"] = np.concatenate([t for _, _, t in scenes])
        s["dts"] = [FIT_DT] * len(scenes)
        return s
    if kind == "gate4":
        p, bonds, _ = create_mpm_gate4_scene(seed=seed % (1 << 32), liquid_particle_diameter=case["diameter"])
        config = create_mpm_gate4_step_config(fracture_bonds=bonds)
        s["solver"] = create_mpm_mls_gpu_solver(p, config)
        s["dt"], s["gravity"] = 1 / 1200, DAM_GRAVITY
    else:
        p, config, s["dt"], s["gravity"] = scene_of(case, seed)
        if kind == "tank":
            s["solver"] = create_mpm_mls_gpu_solver(p, config, TANK_BOUNDS)
        elif case.get("fixed"):
            s["solver"] = create_experimental_mpm_mls_atomic_gpu_solver(p, config, fixed_point_shift=16)
        elif kind == "materials":
            s["solver"] = create_mpm_mls_gpu_solver(p, config)
        else:
            s["solver"] = create_mpm_mls_gpu_solver(p, config, {"waveSpeedBound": DAM_WAVE, "velocityBound": DAM_SPEED})
    if kind == "tank" and case["steps"] == 0:
        s["plan"] = macrostep_plan(case, 1 / 120)
    elif kind == "surface":
        s["plan"] = macrostep_plan(case, 1 / 240)
    if case.get("restart") or kind in ("materials", "gate4"):
        s["start"], _ = s["solver"].read_particles_packed()
    return s


def macrostep_plan(case, macro_dt):
    if case["kind"] == "tank":
        dx, wave, speed = 0.2 / case["side"], TANK_BOUNDS["waveSpeedBound"], TANK_BOUNDS["velocityBound"]
    else:
        dx, wave, speed = 10.0, DAM_WAVE, DAM_SPEED
    return macro_dt, calculate_mpm_cfl_microsteps(macro_dt, dx, wave, speed, NO_LIMIT), speed


def columns(packed, ids):
    return {"position": packed[:, 0:2], "velocity": packed[:, 2:4], "C": packed[:, 4:8], "F": packed[:, 8:12],
            "material": packed[:, 12:20], "object": ids}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "adjoint":
        engine = s["engine"]
        engine.set_velocities(s["velocities"])
        loss = engine.forward(case["steps"], s["dts"], s["targets"], checkpoint_every=case["every"])
        velocities, parameters = engine.backward()
        return {"loss": loss, "velocities": velocities, "parameters": parameters}
    solver = s["solver"]
    if kind == "tanks":
        solver.step_batch(s["steps"], s["dts"], TANK_GRAVITY)
        speeds, _, status = solver.read_compact()
        read = [solver.read_particles_packed(k) for k in range(case["scenes"])]
        return {"status": status[:, 0], "particles": [np.concatenate([p for p, _ in read]),
                                                      np.concatenate([i for _, i in read])]}
    if "start" in s:
        solver.write_particles_packed(s["start"])
    if "plan" in s:
        macro_dt, plan, speed = s["plan"]
        solver.step_cfl_batch(1, macro_dt, plan, speed, NO_LIMIT, s["gravity"])
        most = solver.measure_maximum_particle_speed()["maximumSpeed"]
        if kind == "surface":
            return {"speed": most, "field": solver.gather_surface_occupancy()}
        return dict(columns(*solver.read_particles_packed()), speed=most)
    solver.step_batch(case["steps"], s["dt"], s["gravity"])
    return columns(*solver.read_particles_packed())


# ------------------------------------------------------------------- bounds --

def work(case):
    """Per particle and substep the state is read and written once: 56 + 48 bytes (x, v, C, F, volume and
    material in; x, v, C, F out), and at 2 x 2 particles a cell about a quarter of a node's 64 bytes; about
    400 operations.  Reading the particles back is 84 bytes each, putting them back 80."""
    kind = case["kind"]
    if kind == "adjoint":
        n = case["scenes"] * (case["columns"] * case["rows"] + case["solid"] ** 2)
        # forward: the state in and out; backward: the state and the adjoints in, the adjoints out (the
        # recompute of a checkpointed segment is the price of memory, not of the result)
        return {"bytes": case["steps"] * n * (104.0 + 200.0) + n * 24.0, "flops": case["steps"] * n * 1600.0}
    if kind == "tanks":
        n = case["scenes"] * (case["particles"] - 1000) / math.log(case["particles"] / 1000)
        return {"bytes": n * (120.0 * case["steps"] + 84.0), "flops": n * case["steps"] * 400.0}
    steps = case.get("steps") or macrostep_plan(case, 1 / 120 if kind == "tank" else 1 / 240)[1]["stepCount"]
    n = 3674.0 if kind == "gate4" else case["particles"]
    moved = 84.0 + (80.0 if case.get("restart") or kind in ("materials", "gate4") else 0.0)
    if kind == "surface":
        moved = 36.0 + 8.0 * 1.3 / 4
    return {"bytes": n * (120.0 * steps + moved), "flops": n * steps * 400.0}


# ------------------------------------------- the substep in 64-bit arithmetic --

def det(F):
    return F[:, 0] * F[:, 3] - F[:, 1] * F[:, 2]


def rotation(F):
    a, b = F[:, 0] + F[:, 3], F[:, 2] - F[:, 1]
    r = torch.sqrt(a * a + b * b)
    return torch.stack([a / r, -b / r, b / r, a / r], dim=1)


def mul(A, B):
    return torch.stack([A[:, 0] * B[:, 0] + A[:, 1] * B[:, 2], A[:, 0] * B[:, 1] + A[:, 1] * B[:, 3],
                        A[:, 2] * B[:, 0] + A[:, 3] * B[:, 2], A[:, 2] * B[:, 1] + A[:, 3] * B[:, 3]], dim=1)


def transposed(A):
    return A[:, [0, 2, 1, 3]]


def singular(F):
    """U, (s0, s1), V of F = U diag(s) V^T with s0 >= s1, U and V rotations."""
    u, s, vt = torch.linalg.svd(F.reshape(-1, 2, 2))
    flip = torch.where(torch.linalg.det(u) < 0, -1.0, 1.0)
    u = torch.stack([u[:, :, 0], u[:, :, 1] * flip[:, None]], dim=2)
    vt = torch.stack([vt[:, 0], vt[:, 1] * flip[:, None]], dim=1)
    return u.reshape(-1, 4), s[:, 0], s[:, 1], vt.reshape(-1, 4)


def composed(u, a, b, vt):
    z = torch.zeros_like(a)
    return mul(mul(u, torch.stack([a, z, z, b], dim=1)), vt)


def stress(m, F, plastic, lam, mu):
    """P F^T of one model."""
    J = det(F)
    model = m["model"]
    z = torch.zeros_like(J)
    if model in ("water", "oil"):
        if "equationOfState" in m:
            v = -J * (lam * (torch.pow(1 / J, f32(m["equationOfState"]["exponent"])) - 1))
        else:
            v = lam * torch.clamp(J - 1, max=0.0)
        return torch.stack([v, z, z, v], dim=1)
    one = torch.tensor([1.0, 0.0, 0.0, 1.0], dtype=F.dtype, device=F.device)
    if model == "neo-hookean":
        return mu * (mul(F, transposed(F)) - one) + (lam * torch.log(J))[:, None] * one
    if model == "powder":
        u, s0, s1, _ = singular(F)
        l0, l1 = torch.log(s0), torch.log(s1)
        trace = l0 + l1
        pressure = torch.clamp(-(lam + mu) * torch.clamp(trace, min=math.log(0.5)), min=0.0)
        shear = torch.minimum(0.5 * (l0 - l1), f32(m["frictionCoefficient"]) * pressure / (2 * mu))
        p0, p1 = (2 * mu * (0.5 * trace + d) + lam * trace for d in (shear, -shear))
        return composed(u, p0, p1, transposed(u))
    hard = torch.exp(torch.clamp(10 * (1 - plastic), -20, 20)) if model == "snow" else torch.ones_like(J)
    return (2 * mu * hard)[:, None] * mul(F - rotation(F), transposed(F)) + (lam * hard * J * (J - 1))[:, None] * one


def projected(m, T, plastic):
    """(F, plastic volume) after the model's projection of the trial T."""
    model = m["model"]
    if model in ("water", "oil"):
        return torch.sqrt(torch.clamp(det(T), 0.5, 2.0))[:, None] * rotation(T), plastic
    if model == "snow":
        u, s0, s1, vt = singular(T)
        a, b = torch.clamp(s0, 1 - 0.025, 1 + 0.0075), torch.clamp(s1, 1 - 0.025, 1 + 0.0075)
        return composed(u, a, b, vt), torch.clamp(plastic * det(T) / (a * b), 0.6, 20.0)
    if model == "powder":
        u, s0, s1, vt = singular(T)
        lam, mu = f32(m["lambda"]), f32(m["mu"])
        l0, l1 = torch.log(s0), torch.log(s1)
        trace, least = l0 + l1, math.log(0.5)
        most = f32(m["frictionCoefficient"]) * torch.clamp(-(lam + mu) * torch.clamp(trace, min=least), min=0.0) / (2 * mu)
        shear = 0.5 * (l0 - l1)
        keep = (shear <= most) & (trace >= least)
        mean, shear = 0.5 * torch.clamp(trace, min=least), torch.minimum(shear, most)
        return torch.where(keep[:, None], T, composed(u, torch.exp(mean + shear), torch.exp(mean - shear), vt)), plastic
    return T, plastic  # the neo-hookean stretch limits are far from what these cases reach


class Exact:
    """One scene in 64 bits: x, v, C, F (rows as in the packed record) and plastic volume."""

    def __init__(self, p, config, dt, gravity):
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def t(a):
            return torch.from_numpy(np.asarray(a, np.float32).astype(np.float64)).to(dev)

        self.x, self.v = t(np.stack([p.px, p.py], 1)), t(np.stack([p.vx, p.vy], 1))
        self.C, self.F, self.plastic, self.volume = t(p.C), t(p.F), t(p.plastic_volume), t(p.volume)
        self.materials = list(p.materials) or [config["material"]]
        index = np.maximum(p.material, 0)
        self.of = [torch.from_numpy(np.flatnonzero(index == k)).to(dev) for k in range(len(self.materials))]
        channel = np.array([{"water": 1, "oil": 2}.get(m["model"], 0) for m in self.materials])[index]
        self.channel = torch.from_numpy(channel).to(dev)
        density = np.array([f32(m.get("density", 0.0)) for m in self.materials])[index]
        self.density = torch.from_numpy(density).to(dev)
        self.mass = torch.where(self.channel > 0, self.density * self.volume,
                                torch.full_like(self.volume, f32(config["particleMass"])))
        g = config["grid"]
        self.cells, self.dx = (g["cellsX"], g["cellsY"]), f32(g["cellSize"])
        self.dt, self.g = f32(dt), (f32(gravity["x"]), f32(gravity["y"]))
        self.friction = f32(config.get("wallFriction") or 0.0)
        self.parameters = [(f32(m["lambda"]), f32(m["mu"])) for m in self.materials]
        w, h = self.cells[0] + 3, self.cells[1] + 3
        self.w, self.h = w, h
        n = torch.arange(w * h, device=dev)
        self.nx, self.ny = (n % w - 1).double(), (torch.div(n, w, rounding_mode="floor") - 1).double()

    def by_material(self, f, *arrays):
        """f(material index, rows ...) of each material's particles, put back in order."""
        rows = torch.cat(self.of)
        parts = [f(k, *(a[i] for a in arrays)) for k, i in enumerate(self.of) if i.numel()]
        back = torch.argsort(rows)
        if isinstance(parts[0], tuple):
            return tuple(torch.cat([p[j] for p in parts])[back] for j in range(len(parts[0])))
        return torch.cat(parts)[back]

    def walls(self, u):
        out = []
        for axis, coord, extent in ((0, self.nx, self.cells[0]), (1, self.ny, self.cells[1])):
            c = min(8.0, extent / 4.0)
            a = u[..., axis]
            out.append(a * torch.clamp(torch.where(a < 0, coord, extent - coord) / c, 0.0, 1.0))
        if self.friction > 0:
            for axis, coord, extent in ((0, self.ny, self.cells[1]), (1, self.nx, self.cells[0])):
                c = min(8.0, extent / 4.0)
                near = torch.clamp(torch.minimum(coord, extent - coord), min=0.0)
                out[axis] = out[axis] * (1 - self.friction * (1 - torch.clamp(near / c, 0.0, 1.0)))
        return torch.stack(out, dim=-1)

    def grid(self, sums):
        """Node velocities (channel, node, 2) from the sums (channel, node, (m, px, py, V))."""
        m = sums[..., 0]
        full = m > 0
        u = sums[..., 1:3] / torch.where(full, m, torch.ones_like(m))[..., None]
        u = u + self.dt * torch.tensor(self.g, dtype=u.dtype, device=u.device)
        u = torch.where(full[..., None], u, torch.zeros_like(u))
        W, O = sums[1], sums[2]
        both = ((W[:, 0] > 0) & (O[:, 0] > 0) & (W[:, 3] > 0) & (O[:, 3] > 0) & (self.nx >= 0) & (self.ny >= 0)
                & (self.nx <= self.cells[0]) & (self.ny <= self.cells[1]))
        i = torch.nonzero(both)[:, 0]
        if i.numel():
            vol = torch.nn.functional.pad(sums[1:3, :, 3].reshape(2, self.h, self.w), (1, 1, 1, 1))
            grad = torch.stack([vol[:, 1:-1, 2:] - vol[:, 1:-1, :-2], vol[:, 2:, 1:-1] - vol[:, :-2, 1:-1]], dim=-1)
            grad = grad.reshape(2, -1, 2)[:, i]
            sep = grad[1] - grad[0]
            length = sep.norm(dim=1)
            nrm = sep / torch.clamp(length, min=1e-300)[:, None]
            wd, od = W[i, 0] / W[i, 3], O[i, 0] / O[i, 3]
            contrast = (od - wd) / torch.maximum(wd, od)
            gm = math.hypot(*self.g)
            align = (nrm[:, 0] * self.g[0] + nrm[:, 1] * self.g[1]) / gm if gm > 0 else torch.zeros_like(wd)
            nrm = torch.where((contrast * align < -1e-3)[:, None], -nrm, nrm)
            rel = ((u[2, i] - u[1, i]) * nrm).sum(1)
            overlap = torch.clamp(2 * torch.minimum(W[i, 3], O[i, 3]) / (W[i, 3] + O[i, 3]), 0.0, 1.0)
            least = torch.maximum(0.25 * overlap * self.dx / 0.05, torch.clamp(-rel, min=0.0))
            push = torch.where((length > 1e-8) & (rel < least), (least - rel) / (1 / W[i, 0] + 1 / O[i, 0]), 0.0)
            u = u.clone()
            u[1, i] -= (push / W[i, 0])[:, None] * nrm
            u[2, i] += (push / O[i, 0])[:, None] * nrm
        return self.walls(u)

    def step(self):
        dt, dx, gs = self.dt, self.dx, 4.0 / (self.dx * self.dx)
        liquid = self.channel > 0
        J = det(self.F)
        s = self.by_material(lambda k, F, pv: stress(self.materials[k], F, pv, *self.parameters[k]), self.F, self.plastic)
        A = self.mass[:, None] * self.C - (dt * gs * self.volume)[:, None] * s
        at = self.x / dx
        base = torch.floor(at.detach() - 0.5)
        f = at - base
        weights = [0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2]
        node0 = ((base[:, 1] + 1) * self.w + base[:, 0] + 1).long()
        nodes = self.w * self.h
        sums = torch.zeros(3 * nodes, 4, dtype=f.dtype, device=f.device)
        area = torch.where(liquid, self.volume * J, torch.zeros_like(J))
        around = []
        for oy in range(3):
            for ox in range(3):
                w = weights[ox][:, 0] * weights[oy][:, 1]
                d = torch.stack([ox - f[:, 0], oy - f[:, 1]], dim=1) * dx
                q = self.mass[:, None] * self.v + torch.stack([A[:, 0] * d[:, 0] + A[:, 1] * d[:, 1],
                                                               A[:, 2] * d[:, 0] + A[:, 3] * d[:, 1]], dim=1)
                index = node0 + oy * self.w + ox
                row = torch.cat([(w * self.mass)[:, None], w[:, None] * q, (w * area)[:, None]], dim=1)
                sums = sums.index_add(0, self.channel * nodes + index, row)
                around.append((w, d, index))
        sums = sums.reshape(3, nodes, 4)
        u = self.grid(sums).reshape(3 * nodes, 2)
        total = sums[1] + sums[2]
        v, B = torch.zeros_like(self.v), torch.zeros_like(self.C)
        pm, pv = torch.zeros_like(J), torch.zeros_like(J)
        for w, d, index in around:
            wu = w[:, None] * u[self.channel * nodes + index]
            v = v + wu
            B = B + torch.stack([wu[:, 0] * d[:, 0], wu[:, 0] * d[:, 1], wu[:, 1] * d[:, 0], wu[:, 1] * d[:, 1]], dim=1)
            pm, pv = pm + w * total[index, 0], pv + w * total[index, 3]
        one = torch.ones_like(J)
        pd, ld = torch.where(liquid, self.density, one) / J, torch.where(liquid, pm, one) / torch.where(liquid, pv, one)
        rd = torch.where(liquid, (pd - ld) / pd, torch.zeros_like(J))
        v = v + dt * rd[:, None] * torch.tensor(self.g, dtype=v.dtype, device=v.device)
        C = B * gs
        x = self.x + dt * v
        row = torch.maximum(C[:, 0].abs() + C[:, 1].abs(), C[:, 2].abs() + C[:, 3].abs()).detach()
        n = torch.clamp(torch.ceil(dt * row * 4.0), min=1.0)
        h = (dt / n)[:, None]
        U = torch.tensor([1.0, 0.0, 0.0, 1.0], dtype=C.dtype, device=C.device) + h * C
        T = self.F
        for k in range(int(n.max().item())):
            T = torch.where((n > k)[:, None], mul(U, T), T)
        self.F, self.plastic = self.by_material(lambda k, t, pl: projected(self.materials[k], t, pl), T, self.plastic)
        most = torch.tensor([self.cells[0] * self.dx, self.cells[1] * self.dx], dtype=x.dtype, device=x.device)
        out = (x < 0) | (x > most) | ((x == 0) & (v < 0)) | ((x == most) & (v > 0))
        self.v = torch.where(out, torch.zeros_like(v), v)
        self.x = torch.where(x < 0, torch.zeros_like(x), torch.where(x > most, most.expand_as(x), x))
        self.C = C

    def field(self):
        """Water and oil display area 2 V J w / dx^2 of every halo node."""
        at = self.x / self.dx
        base = torch.floor(at - 0.5)
        f = at - base
        weights = [0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2]
        out = torch.zeros(self.w * self.h * 2, dtype=f.dtype, device=f.device)
        area = 2 * self.volume * det(self.F) / self.dx ** 2
        for oy in range(3):
            for ox in range(3):
                node = ((base[:, 1] + 1 + oy) * self.w + base[:, 0] + 1 + ox).long()
                out.index_add_(0, node * 2 + self.channel - 1, weights[ox][:, 0] * weights[oy][:, 1] * area)
        return out.reshape(self.h, self.w, 2).cpu().numpy()

    def columns(self):
        return {"position": self.x.cpu().numpy(), "velocity": self.v.cpu().numpy(), "C": self.C.cpu().numpy(),
                "F": self.F.cpu().numpy(), "material": None, "object": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "gate4":
        return None  # its bonded edges turn the rounding of a position into a velocity by 1 / dt
    if kind == "adjoint":
        n = case["scenes"] * (case["columns"] * case["rows"] + case["solid"] ** 2)
        if n * case["steps"] > 5_000_000 or case["steps"] > 100:
            return None  # the gradient of a long trajectory takes minutes
        losses, velocities, parameters = [], [], []
        for k in range(case["scenes"]):
            p, config, targets = fit_scene(case, np.random.default_rng([seed, 31, k]))
            e = Exact(p, config, FIT_DT, DAM_GRAVITY)
            v0 = e.v.requires_grad_(True)
            theta = torch.tensor([f32(ADJOINT_WATER["lambda"]), f32(ADJOINT_SOLID["lambda"]), f32(ADJOINT_SOLID["mu"])],
                                 dtype=torch.float64, device=v0.device, requires_grad=True)
            e.v = v0
            e.parameters = [(theta[0], 0.0), (theta[1], theta[2])]
            for _ in range(case["steps"]):
                e.step()
            loss = ((e.x - torch.from_numpy(targets.astype(np.float64)).to(v0.device)) ** 2).sum()
            loss.backward()
            losses.append(float(loss.detach()))
            velocities.append(v0.grad.cpu().numpy())
            parameters.append(theta.grad.cpu().numpy())
        return {"loss": np.array(losses), "velocities": np.concatenate(velocities), "parameters": np.stack(parameters)}
    if kind == "tanks":
        rows = []
        for p, config in tank_scenes(case, seed):
            e = Exact(p, config, 0.3 * config["grid"]["cellSize"] / 33.0, TANK_GRAVITY)
            for _ in range(case["steps"]):
                e.step()
            c = e.columns()
            n = len(p)
            m = TAIT
            fixed = np.tile([m["lambda"], 0.0, m["density"], f32(config["particleVolume"]), 7.0, 0.0], (n, 1))
            code = np.full((n, 1), float(np.array(2, np.uint32).view(np.float32)))  # the model's bits
            rows.append(np.hstack([c["position"], c["velocity"], c["C"], c["F"], np.ones((n, 1)), code, fixed]))
        return {"status": None, "particles": [np.concatenate(rows), None]}
    p, config, dt, gravity = scene_of(case, seed)
    steps = case.get("steps")
    if not steps:
        plan = macrostep_plan(case, 1 / 120 if kind == "tank" else 1 / 240)[1]
        steps, dt = plan["stepCount"], plan["microDt"]
    e = Exact(p, config, dt, gravity)
    for _ in range(steps):
        e.step()
    speed = float(e.v.norm(dim=1).max())
    if kind == "surface":
        return {"speed": speed, "field": e.field()}
    out = e.columns()
    if "steps" in case and case["steps"] == 0:
        out["speed"] = speed
    return out
