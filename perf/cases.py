"""The work that programs have this framework do, as cases that can be timed.

A case names a path through the public Python binding (`pbf`, `pbf_autograd`)
and its sizes; `prepare` makes what a program has in hand before the call,
`run` is one pass of the call, and `exact` restates the passes' arithmetic in
64 bits with plain torch.

kinds of case
  frame    one frame of one scene in a host loop: the state goes up from
           page-locked buffers, the substeps run, positions and velocities
           come back, and the host waits once.
  batch    the same frame over many scenes held in one particle array.
  rollout  one optimisation step of the differentiable rollout: forward,
           loss, backward, through the torch function.
  render   one image of the particles, read back.
  sort     keys, stable sort and cell table of device positions through the
           entry point for hosts that may not allocate.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "position-based-fluids_gb300"))
import pbf  # noqa: E402
import pbf_autograd  # noqa: E402


def listed():
    return [
        # the smallest scene that the repository steps (its smoke check): launches and latency count
        {"name": "frame_2k", "kind": "frame", "scene": "block", "n": 2048, "iterations": 4, "substeps": 2, "warm": 50,
         "mode": "exact", "grid": 0, "tune": False},
        # the small dam break, the scene a new user starts from
        {"name": "frame_32k", "kind": "frame", "scene": "block", "n": 32768, "iterations": 4, "substeps": 2,
         "warm": 50, "mode": "exact", "grid": 0, "tune": False},
        # an odd count, an odd iteration count and a hash size that is no power of two
        {"name": "frame_99991_odd", "kind": "frame", "scene": "double", "n": 99991, "iterations": 3, "substeps": 1,
         "warm": 30, "mode": "exact", "grid": 300007, "tune": False},
        # the particle-count sweep's smallest entry
        {"name": "frame_262k_i2", "kind": "frame", "scene": "double", "n": 262144, "iterations": 2, "substeps": 2,
         "warm": 30, "mode": "exact", "grid": 0, "tune": False},
        # the benchmark's dam break in the middle of its collapse, tuned as the benchmark tunes it
        {"name": "frame_1m", "kind": "frame", "scene": "block", "n": 1048576, "iterations": 4, "substeps": 2,
         "warm": 50, "mode": "exact", "grid": 0, "tune": True},
        # the same scene in the relaxed arithmetic, with the default launch shape, read back every substep
        {"name": "frame_1m_relaxed", "kind": "frame", "scene": "block", "n": 1048576, "iterations": 4, "substeps": 1,
         "warm": 50, "mode": "relaxed", "grid": 0, "tune": False},
        # physically complete neighbour sets: the longest friend lists that are walked
        {"name": "frame_131k_complete", "kind": "frame", "scene": "block", "n": 131072, "iterations": 4,
         "substeps": 2, "warm": 20, "mode": "complete", "grid": 0, "tune": False},
        # the sweep's largest entry
        {"name": "frame_8m", "kind": "frame", "scene": "double", "n": 8388608, "iterations": 4, "substeps": 2,
         "warm": 10, "mode": "exact", "grid": 0, "tune": False},
        # many small scenes with their own boxes, gravity and viscosity (a data-generation batch)
        {"name": "batch_64", "kind": "batch", "scenes": 64, "sizes": 7, "iterations": 4, "substeps": 2, "warm": 50},
        # a gradient step on gravity, viscosity and initial velocities
        {"name": "rollout_65k", "kind": "rollout", "nx": 64, "ny": 32, "nz": 32, "substeps": 20, "every": 10},
        # a preview image at the scale of the reference's scenes
        {"name": "render_262k", "kind": "render", "n": 262144, "width": 1280, "height": 720},
        # the sort stage alone, for hosts that own their device memory
        {"name": "sort_1000003", "kind": "sort", "n": 1000003, "grid": 1 << 19},
    ]


def draw(rng):
    kind = rng.choice(["frame"] * 7 + ["batch", "rollout", "render", "sort"])

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "frame":
        n = log_int(2048, 3000000)
        mode = rng.choice(["exact", "exact", "exact", "relaxed", "complete"])
        grid = rng.choice([0, 0, 0, log_int(max(1024, n // 2), 4 * n) | 1])
        return {"kind": kind, "scene": rng.choice(["block", "double"]), "n": n, "iterations": rng.randint(2, 8),
                "substeps": rng.randint(1, 3), "warm": rng.randint(5, 50) if n < 1500000 else rng.randint(2, 10),
                "mode": mode, "grid": grid, "tune": rng.random() < 0.25}
    if kind == "batch":
        return {"kind": kind, "scenes": log_int(4, 96), "sizes": rng.randint(1, 1000), "iterations": rng.randint(2, 6), "substeps": rng.randint(1, 3),
                "warm": rng.randint(5, 50)}
    if kind == "rollout":
        return {"kind": kind, "nx": rng.randint(16, 72), "ny": rng.randint(12, 36), "nz": rng.randint(12, 36),
                "substeps": rng.randint(6, 20), "every": rng.randint(4, 10)}
    if kind == "render":
        return {"kind": kind, "n": log_int(8192, 600000), "width": rng.randint(320, 1600),
                "height": rng.randint(240, 1000)}
    return {"kind": "sort", "n": log_int(3000, 1048576), "grid": rng.choice([1 << rng.randint(12, 20),
                                                                           log_int(5000, 900000)])}


# ------------------------------------------------------------ the scenes --
SPACING, ORIGIN, JITTER = 0.05, (0.025, 0.025, 0.025), 0.005


def _block_scene(n, iterations, seed):
    """A dam-break block of n particles (2:1:2, as the benchmark's, cut at n)
    in a box twice as long as the block, with the benchmark's solver settings."""
    ny = max(1, round((n / 4.0) ** (1.0 / 3.0)))
    nx = nz = 2 * ny
    while nx * ny * nz < n:
        nz += 1
    pos = pbf.scene_block(nx, ny, nz, SPACING, ORIGIN, JITTER, seed)[:n].copy()
    params = pbf.load_scenario("dam_break_1m")
    params.particleCount, params.simIterations = n, iterations
    box = (0.0, 2 * nx * SPACING, 0.0, 2 * ny * SPACING, 0.0, nz * SPACING)
    params.xMin, params.xMax, params.yMin, params.yMax, params.zMin, params.zMax = box
    params.gridBufSize = pbf.grid_size_for_box(box, params.h)
    return params, pos, np.zeros_like(pos)


def _scene(case, seed):
    if case["scene"] == "block":
        params, pos, vel = _block_scene(case["n"], case["iterations"], seed)
    else:
        params, pos, vel = pbf.make_double_dam_break(case["n"], case["iterations"], seed)
    if case["grid"]:
        params.gridBufSize = case["grid"]
    params.completeNeighbours = int(case["mode"] == "complete")
    return params, pos, vel


def _pinned(n):
    return torch.empty((n, 4), dtype=torch.float32, pin_memory=True)


def _frame_state(case, sim):
    """The host side of a frame loop: the running state in page-locked
    buffers, and the buffers that the next frame's state comes back to."""
    state = {"case": case, "sim": sim, "substeps": case["substeps"]}
    for name in ("pos", "vel", "out_pos", "out_vel"):
        state[name] = _pinned(sim.n)
    sim.read_state_into(state["pos"].data_ptr(), state["vel"].data_ptr())
    return state


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frame":
        params, pos, vel = _scene(case, seed)
        sim = pbf.Simulation.create(params, pos, vel)
        sim.Step(2 * case["warm"])  # into the collapse: compressed, with splashes
        if case["mode"] == "relaxed":
            params.relaxedMath = 1
            sim.set_params(params)
        if case["tune"]:
            sim.autotune()
        return {**_frame_state(case, sim), "scenes": [params]}
    if kind == "batch":
        scenes, positions = pbf.make_batch_scenes(case["scenes"], case["sizes"])
        for p in scenes:
            p.simIterations = case["iterations"]
        pos = np.concatenate(positions)
        vel = np.zeros_like(pos)
        vel[:, :3] = np.random.default_rng(seed).normal(0.0, 0.05, (len(pos), 3))
        sim = pbf.Simulation.create(scenes, pos, vel)
        sim.Step(2 * case["warm"])
        return {**_frame_state(case, sim), "scenes": scenes}
    if kind == "rollout":
        params, pos, vel = pbf.make_rollout_scene(case["nx"], case["ny"], case["nz"], seed)
        rng = np.random.default_rng(seed)
        v0 = torch.from_numpy(rng.normal(0.0, 0.05, (len(pos), 3)).astype(np.float32))
        sim = pbf.Simulation.create(pbf.rollout_target_params(params), pos, vel)
        sim.Step(case["substeps"])
        target = torch.from_numpy(sim.positions_by_id()[:, :3].copy())
        sim.set_params(params)
        return {"case": case, "sim": sim, "params": params, "x0": pos, "v0": v0, "target": target,
                "visc": torch.tensor(float(params.viscosityFactor)),
                "gravity": torch.tensor([params.gravityX, params.gravityY, params.gravityZ])}
    if kind == "render":
        side = 1  # smoothing length 2 and spacing 0.55, as in the reference's scenes: a density surface to shade
        while side ** 3 < case["n"]:
            side += 1
        params = pbf.load_scenario("dam_break_32k")
        params.particleCount, params.h, params.h_2 = case["n"], 2.0, 4.0
        pos = pbf.scene_block(side, side, side, 0.55, (0.3, 0.3, 0.3), 0.05, seed)[:case["n"]].copy()
        pos[:, 3] = np.random.default_rng(seed).uniform(0.0, 40.0, len(pos))  # speeds
        sim = pbf.Simulation.create(params, pos, np.zeros_like(pos))
        size = 0.55 * side
        cam = pbf.render_camera((0.5 * size, 0.9 * size, 2.7 * size), (0.5 * size, 0.45 * size, 0.5 * size),
                                (0.0, 1.0, 0.0), 45.0, case["width"], case["height"], 1.0)
        return {"case": case, "sim": sim, "cam": cam}
    params, pos, _ = _block_scene(case["n"], 4, seed)
    params.gridBufSize = case["grid"]
    rng = np.random.default_rng(seed)
    pos[:, :3] += rng.uniform(-0.04, 0.04, (len(pos), 3)).astype(np.float32)
    pred = torch.from_numpy(pos).cuda()
    ints = [torch.empty(k, dtype=torch.int32, device="cuda") for k in (case["n"], case["n"], 2 * case["grid"])]
    return {"case": case, "params": params, "pred": pred, "keys": ints[0], "perm": ints[1], "cells": ints[2]}


def run(state):
    kind = state["case"]["kind"]
    if kind in ("frame", "batch"):
        sim = state["sim"]
        sim.write_state_async(state["pos"].data_ptr(), state["vel"].data_ptr())
        sim.step_read_async(state["substeps"], state["out_pos"].data_ptr(), state["out_vel"].data_ptr())
        sim.synchronize()
        return {"pos": state["out_pos"], "vel": state["out_vel"]}
    if kind == "rollout":
        case = state["case"]
        v0 = state["v0"].clone().requires_grad_()
        visc = state["visc"].clone().requires_grad_()
        gravity = state["gravity"].clone().requires_grad_()
        x = pbf_autograd.rollout(v0, visc, gravity, state["sim"], state["params"], state["x0"], case["substeps"],
                                 case["every"])
        loss = 0.5 * (x - state["target"]).square().sum()
        loss.backward()
        return {"x": x.detach(), "dv0": v0.grad, "dvisc": visc.grad, "dgravity": gravity.grad}
    if kind == "render":
        sim, cam = state["sim"], state["cam"]
        sim.render_frame(cam, 0)
        return {"image": sim.render_read(cam, 0)}
    pbf.sort_state_noalloc(state["params"], state["pred"].data_ptr(), state["keys"].data_ptr(),
                           state["perm"].data_ptr(), state["cells"].data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
    return {"keys": state["keys"], "perm": state["perm"], "cells": state["cells"]}


def work(case):
    """Bytes: inputs read once, outputs written once.  Operations: those of
    the friends' contributions, at the mean list lengths of a running scene
    (28 friends in the density pass, 24 in the others, 55 within h)."""
    kind = case["kind"]
    if kind in ("frame", "batch"):
        n = case["n"] if kind == "frame" else case["scenes"] * 22000
        dense, other = (55, 55) if case.get("mode") == "complete" else (28, 24)
        pairs = 55 * 9 + case["iterations"] * (28 * dense + 30 * other) + (36 + 28) * other
        return {"bytes": 64 * n, "flops": case["substeps"] * n * pairs}
    if kind == "rollout":
        n = case["nx"] * case["ny"] * case["nz"]
        pairs = 55 * 9 + 4 * (28 * 22 + 30 * 19) + (36 + 28) * 19
        return {"bytes": 64 * n, "flops": 3 * case["substeps"] * n * pairs}
    if kind == "render":
        return {"bytes": 16 * case["n"] + 16 * case["width"] * case["height"], "flops": 100 * case["width"] * case["height"]}
    return {"bytes": 24 * case["n"] + 8 * case["grid"], "flops": 40 * case["n"]}


# ------------------------------------------------- the passes in 64 bits --
# What is decided rather than computed (the cells, the friend lists with their
# circles, limits and order) is decided in 32 bits, as the framework's
# contract has it; every sum and quotient is in 64 bits.
def _six_digits(v):
    return float(np.float32(float("%.6g" % v)))


def _spread(x):
    x = x & 0xFFFFFFFF
    for shift, mask in ((16, 0x030000FF), (8, 0x0300F00F), (4, 0x030C30C3), (2, 0x09249249)):
        x = (x | (x << shift)) & mask
    return x


def _hash(c, grid):
    return (_spread(c[..., 0]) | (_spread(c[..., 1]) << 1) | (_spread(c[..., 2]) << 2)) % grid


def _one(value, dev):
    """A 32-bit value on the device: torch divides by it, where by a plain number it multiplies by the reciprocal."""
    return torch.tensor(float(value), dtype=torch.float32, device=dev)


def _friends(q, cell, key, params, rows):
    """The friends of the particles `rows`: (particle, friend, circle) in list order, without those over a circle's limit."""
    C, dev, grid = int(params.friendsCircles), q.device, int(params.gridBufSize)
    o = torch.tensor([(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)], device=dev)
    want = _hash(cell[rows][:, None, :] + o, grid)
    lo, hi = torch.searchsorted(key, want), torch.searchsorted(key, want, right=True)
    count = (hi - lo).reshape(-1)
    i = rows.repeat_interleave((hi - lo).sum(1))
    at = torch.arange(len(i), device=dev) - (count.cumsum(0) - count).repeat_interleave(count)
    j = lo.reshape(-1).repeat_interleave(count) + at
    r = q[i] - q[j]
    r2 = (r[:, 0] * r[:, 0] + r[:, 1] * r[:, 1]) + r[:, 2] * r[:, 2]
    # its own entry is left out; under a hash collision a cell can be met twice, and each time counts
    same = (want == key[rows][:, None]).reshape(-1).repeat_interleave(count)
    take = (r2 < float(params.h_2)) & ~((i == j) & same)
    i, j, r2 = i[take], j[take], r2[take]
    lo_r = np.float32(0.3) * np.float32(params.h)
    adj = ((r2.sqrt() - float(lo_r)) / _one(np.float32(params.h) - lo_r, dev)).clamp_min(0.0)
    circle = (adj * adj * adj * C).to(torch.int64).clamp_max(C - 1)
    group = i * C + circle
    order = torch.sort(group, stable=True).indices
    i, j, circle, group = i[order], j[order], circle[order], group[order]
    first = torch.searchsorted(group, group)
    take = torch.arange(len(i), device=dev) - first < int(params.particlesPerCircle)
    return i[take], j[take], circle[take]


def _structure(q, params):
    """Sort order of the predictions q (32 bits) and the pairs of the density pass and of the others."""
    n, dev, C = len(q), q.device, int(params.friendsCircles)
    cell = (q / _one(params.h, dev)).to(torch.int64)
    key, perm = torch.sort(_hash(cell, int(params.gridBufSize)), stable=True)
    q, cell = q[perm], cell[perm]
    parts = []
    for a in range(0, n, 32768):
        i, j, circle = _friends(q, cell, key, params, torch.arange(a, min(n, a + 32768), device=dev))
        local = i - a
        m = min(n, a + 32768) - a
        counts = torch.bincount(local * C + circle, minlength=m * C).reshape(m, C)
        total = counts.sum(1).to(torch.float32)
        before = torch.zeros_like(counts[:, 0])
        keep = []
        for limit in (0.6, 0.5):
            before, kept, open_ = before * 0, torch.zeros_like(counts[:, 0]), torch.ones_like(counts[:, 0], dtype=torch.bool)
            for k in range(C):
                open_ = open_ & ~((before.to(torch.float32) / total) > float(np.float32(limit)))
                kept = torch.where(open_, k + 1, kept)
                before = before + torch.where(open_, counts[:, k], 0)
            keep.append(torch.ones_like(circle, dtype=torch.bool) if params.completeNeighbours else circle < kept[local])
        parts.append((i[keep[0]], j[keep[0]], i[keep[1]], j[keep[1]]))
    i0, j0, i1, j1 = (torch.cat(p) for p in zip(*parts))
    return perm, (i0, j0), (i1, j1)


def _substep64(x, v, gravity, visc, params):
    """One substep of (x, v) in 64 bits: the new x, |v| before viscosity, the new v, and the sort order."""
    dt, h, h2 = float(params.timeStep), float(params.h), float(params.h_2)
    poly6 = _six_digits(315.0 / (64.0 * math.pi * h ** 9))
    grad = _six_digits(45.0 / (math.pi * h ** 6))
    rho0, eps, K = float(params.restDensity), float(params.epsilon), float(params.surfaceTenstionK)
    w_q = (h2 - (float(params.surfaceTenstionDist) * h) ** 2) ** 3
    lo = torch.tensor([params.xMin, params.yMin, params.zMin], dtype=x.dtype, device=x.device)
    hi = torch.tensor([params.xMax, params.yMax, params.zMax], dtype=x.dtype, device=x.device)
    x32, v32, g32 = (t.detach().to(torch.float32) for t in (x, v, gravity))
    perm, dense, other = _structure(x32 + dt * (v32 + dt * g32), params)
    v = v + dt * gravity
    p = x + dt * v
    x, p, n = x[perm], p[perm], len(x)

    def pair(p, ij):
        i, j = ij
        r = p[i] - p[j]
        r2 = r.square().sum(1)
        take = r2.detach() < h2
        if params.zeroDistanceGuard:
            take = take & (r2.detach() > 0)
        i, j, r, r2 = i[take], j[take], r[take], r2[take]
        length = r2.sqrt()
        return i, j, r2, (h - length).square()[:, None] * r / length[:, None]

    def add(i, values):
        return torch.zeros((n, *values.shape[1:]), dtype=values.dtype, device=values.device).index_add(0, i, values)

    rho = None
    for _ in range(int(params.simIterations)):
        i, j, r2, k = pair(p, dense)
        g = grad * k
        rho = poly6 * (add(i, (h2 - r2) ** 3) + (h2 ** 3 if params.completeNeighbours else 0.0))
        norm = add(i, g.square().sum(1)) + add(i, g).square().sum(1)
        lam = -(rho / rho0 - 1.0) / (norm / rho0 ** 2 + eps)
        i, j, r2, k = pair(p, other)
        a = lam[i] + lam[j] + K * ((h2 - r2) ** 3 / w_q) ** 4
        p = p - grad / rho0 * add(i, a[:, None] * k)
        if params.boxClamp:
            p = torch.minimum(torch.maximum(p, lo), hi)
    v = (p - x) / dt
    speed = v.square().sum(1).sqrt()
    i, j, r2, k = pair(p, other)
    if rho is not None:
        take = rho.detach()[j].abs() > 1e-8
        i, j, r2, k = i[take], j[take], r2[take], k[take]
    u = v[j] - v[i]
    omega = -grad * add(i, torch.linalg.cross(u, k))
    w = v + visc * poly6 * add(i, u * ((h2 - r2) ** 3)[:, None])
    square = omega.square().sum(1)
    size = torch.where(square > 0, torch.where(square > 0, square, 1.0).sqrt(), 0.0)
    eta = -grad * add(i, size[j][:, None] * k)
    square = eta.square().sum(1, keepdim=True)
    eta = torch.where(square > 0, eta / torch.where(square > 0, square, 1.0).sqrt(), eta)
    w = w + dt * float(params.vorticityFactor) * torch.linalg.cross(eta, omega)
    return p, speed, w, perm


def _gravity(params, dev):
    g = (params.gravityX, params.gravityY, params.gravityZ) if params.gravityVectorEnable else (0.0, -params.garvity, 0.0)
    return torch.tensor(g, dtype=torch.float64, device=dev)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] in ("frame", "batch"):
        # From the second substep on, a particle that 64 bits put across a cell's face shifts the records behind it
        # in the sort, and the more particles, the more of them there are.
        if case.get("n", 0) > (1200000 if case["substeps"] == 1 else 140000):
            return None
        state = prepare(case, seed)
        pos, vel, at = [], [], 0
        for params in state["scenes"]:
            n = int(params.particleCount)
            x = state["pos"][at:at + n, :3].to(dev, torch.float64)
            v = state["vel"][at:at + n, :3].to(dev, torch.float64)
            at += n
            for _ in range(case["substeps"]):
                x, speed, v, _ = _substep64(x, v, _gravity(params, dev), float(params.viscosityFactor), params)
            pos.append(torch.cat([x, speed[:, None]], 1))
            vel.append(torch.cat([v, torch.zeros_like(speed)[:, None]], 1))
        return {"pos": torch.cat(pos), "vel": torch.cat(vel)}
    if case["kind"] == "rollout":
        state = prepare(case, seed)
        params = state["params"]
        x = torch.from_numpy(state["x0"][:, :3]).to(dev, torch.float64)
        v0 = state["v0"].to(dev, torch.float64).requires_grad_()
        visc = state["visc"].to(dev, torch.float64).requires_grad_()
        gravity = state["gravity"].to(dev, torch.float64).requires_grad_()
        v, ids = v0, torch.arange(len(x), device=dev)
        for _ in range(case["substeps"]):
            # the sort and the friends are taken anew in the backward's recomputation, from the same values
            x, _, v, perm = torch.utils.checkpoint.checkpoint(
                lambda x, v, g, c: _substep64(x, v, g, c, params), x, v, gravity, visc, use_reentrant=False,
                determinism_check="none")
            ids = ids[perm]
        out = torch.zeros_like(x).index_copy(0, ids, x)
        (0.5 * (out - state["target"].to(dev, torch.float64)).square().sum()).backward()
        # over more substeps the paths part: the collapse is chaotic, and the gradients feel it first
        if case["substeps"] > 10:
            return {"x": out.detach(), "dv0": None, "dvisc": None, "dgravity": None}
        return {"x": out.detach(), "dv0": v0.grad, "dvisc": visc.grad, "dgravity": gravity.grad}
    return None
