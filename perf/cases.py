"""The work a program has this framework do, as cases that can be timed one by one.

A case is a dict of plain values; prepare() makes what a program holds before the call (a world with its bodies, or
arrays), run() is one pass through the public entry points and returns its outputs whole.

Kinds:
  substep   bl_gpu_substep_noalloc: one substep of one beam body in the caller's own device buffers (an engine that
            owns its memory, or steps inside its own capture) - the smallest call
  vehicle   World.step_substeps of one vehicle: the truss car at the wall, or a car on driven wheels with shocks
  pair      the same of two trusses with collision skins crashing into each other
  fleet     the same of many vehicles on a heightfield: driving ("grid") or crashing in head-on pairs ("pairs")
  ladder, plate, shell   the implicit step of FEM frames: members alone, a shell plate, a car body of welded panels
  network   the learned warm start's network on host arrays: its forward or its loss gradient

The explicit worlds (vehicle, pair, fleet) start every pass from one stored node state, as rollouts from a stored state
do: the pass copies it into the world's device-resident nodes, steps a frame, and the nodes are its output. The FEM
worlds go on from frame to frame. The program has one stream for all its work, as one that steps one world does: a
frame follows the frame before.
"""
from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

from beamlab_b200 import BEAM_DTYPE, NODE_DTYPE, SoftBody, World, WorldSettings, _lib, rigs, world_from_rig

FRAME = 33  # a 60 Hz frame of 2 kHz substeps
GRAVITY = (0.0, -9.81, 0.0)
DT = 0.0005


def listed():
    return [
        # one substep of the 20 x 4 x 5 truss car's body: two launches, all latency
        {"name": "substep_truss", "kind": "substep", "nx": 20, "ny": 4, "nz": 5},
        # the truss car (400 nodes, 3,121 beams) as its front meets the wall: one vehicle, one frame
        {"name": "truss_car", "kind": "vehicle", "rig": "truss", "nx": 20, "ny": 4, "nz": 5, "warm": 8, "substeps": FRAME},
        # a car on four driven wheels with progressive shocks, rolling on grass (tyres, shocks, drive)
        {"name": "wheeled_car", "kind": "vehicle", "rig": "wheeled", "nx": 14, "ny": 3, "nz": 5, "warm": 12, "substeps": FRAME},
        # two trusses crashing head on: islands, pair search, narrow phase, response
        {"name": "crash_pair", "kind": "pair", "nx": 12, "ny": 4, "nz": 5, "hull": False, "warm": 2, "substeps": FRAME},
        # 64 vehicles driving over the heightfield, few of them touching
        {"name": "fleet64_driving", "kind": "fleet", "vehicles": 64, "layout": "grid", "warm": 16, "substeps": FRAME},
        # the batched fleet of the benchmark at its crash peak: 0.94 M nodes, 8.9 M beams, 128 head-on pairs
        {"name": "fleet256_crashing", "kind": "fleet", "vehicles": 256, "layout": "pairs", "warm": 5, "substeps": FRAME},
        # a ladder frame of members (two rails of 41 nodes), clamped at one end
        {"name": "ladder", "kind": "ladder", "rails": 41, "substeps": FRAME},
        # the 21 x 21-node shell plate, clamped at one edge under a point load
        {"name": "plate21", "kind": "plate", "n": 20, "substeps": FRAME},
        # the 64 x 64-node, 7,938-triangle plate
        {"name": "plate64", "kind": "plate", "n": 63, "substeps": FRAME},
        # a shell car body of about 10 k nodes, eight substeps
        {"name": "shell10k", "kind": "shell", "target": 10000, "substeps": 8},
        # the 50,442-node shell car body, four substeps
        {"name": "shell50k", "kind": "shell", "target": 50000, "substeps": 4},
        # one loss gradient of the warm start's network on the samples of two substeps of the 10 k body
        {"name": "network_gradient", "kind": "network", "op": "gradient", "samples": 20660},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(("substep", "vehicle", "pair", "fleet", "ladder", "plate", "plate", "shell", "shell", "network"))
    if kind == "substep":
        return {"kind": kind, "nx": _log(rng, 4, 60), "ny": rng.randint(2, 7), "nz": rng.randint(2, 9)}
    if kind == "vehicle":
        rig = rng.choice(("truss", "wheeled"))
        return {"kind": kind, "rig": rig, "nx": _log(rng, 8, 40), "ny": rng.randint(3, 6), "nz": rng.randint(4, 8),
                "warm": 8 if rig == "truss" else 12, "substeps": FRAME}
    if kind == "pair":
        return {"kind": kind, "nx": _log(rng, 8, 30), "ny": rng.randint(3, 6), "nz": rng.randint(4, 7),
                "hull": rng.random() < 0.5, "warm": rng.randint(2, 4), "substeps": FRAME}
    if kind == "fleet":
        layout = rng.choice(("grid", "pairs"))
        return {"kind": kind, "vehicles": _log(rng, 4, 96), "layout": layout, "warm": 16 if layout == "grid" else rng.randint(3, 8),
                "substeps": FRAME}
    if kind == "ladder":
        return {"kind": kind, "rails": _log(rng, 6, 120), "substeps": FRAME}
    if kind == "plate":
        return {"kind": kind, "n": _log(rng, 8, 63), "substeps": FRAME}
    if kind == "shell":
        return {"kind": kind, "target": _log(rng, 2000, 30000), "substeps": 4}
    return {"kind": kind, "op": rng.choice(("forward", "gradient")), "samples": _log(rng, 300, 60000)}


# ------------------------------------------------------------------------------------------ inputs
def _dims(case):
    return case["nx"], case["ny"], case["nz"]


@functools.lru_cache(maxsize=2)
def _fleet(vehicles, layout):
    return rigs.fleet(vehicles, seed=3, layout=layout)


def _rig(case, seed):
    kind, dims = case["kind"], None
    rng = np.random.default_rng(seed)
    if kind == "vehicle":
        dims = _dims(case)
        if case["rig"] == "truss":
            return rigs.truss_car(seed, speed=float(rng.uniform(14.0, 16.0)), dims=dims)
        return rigs.wheeled_car(seed, speed=float(rng.uniform(10.0, 14.0)), yaw=float(rng.uniform(0.1, 0.4)), dims=dims,
                                shocks=rigs.SHOCK_TYPES[2])
    if kind == "pair":
        return rigs.crash_pair(seed, speed_a=float(rng.uniform(11.0, 13.0)), speed_b=float(rng.uniform(11.0, 13.0)),
                               hull=case["hull"], dims=_dims(case))
    if kind == "fleet":
        # one fleet's lattices, with stiffnesses and node velocities of the seed
        base = _fleet(case["vehicles"], case["layout"])
        bodies = []
        for b in base["bodies"]:
            b = dict(b)
            b["k"] = (b["k"] * rng.uniform(0.9, 1.1, len(b["k"])).astype(np.float32)).astype(np.float32)
            b["vel"] = (b["vel"] + rng.uniform(-0.02, 0.02, b["vel"].shape)).astype(np.float32)
            bodies.append(b)
        return dict(base, bodies=bodies)
    if kind == "ladder":
        return rigs.frame_ladder(rails=case["rails"], spacing=min(0.25, 6.0 / case["rails"]), load=float(rng.uniform(100.0, 300.0)))
    if kind == "plate":
        return rigs.shell_plate(case["n"], seed=seed)
    return rigs.shell_body(case["target"], seed=seed)


@functools.lru_cache(maxsize=1)
def _stream():
    return torch.cuda.Stream()


class _DeviceNodes:
    """The world's device-resident node array (World.device_nodes) for torch.as_tensor."""

    def __init__(self, world):
        ptr, n = world.device_nodes()
        self.world = world
        self.__cuda_array_interface__ = {"shape": (n, 8), "typestr": "<f4", "data": (ptr, False), "version": 3}


def _incidence(beams, n):
    """Each node's beams in beam order; bit 31 marks the node as the beam's b end."""
    m = len(beams)
    node = np.concatenate([beams["a"], beams["b"]]).astype(np.int64)
    word = np.concatenate([np.arange(m), np.arange(m) | 0x80000000]).astype(np.uint32)
    order = np.lexsort((np.concatenate([np.arange(m), np.arange(m)]), node))
    ptr = np.zeros(n + 1, np.int32)
    ptr[1:] = np.cumsum(np.bincount(node, minlength=n))
    return ptr, word[order].view(np.int32)


def _truss(case, seed):
    """One lattice cantilever (its first slice anchored) with stiffnesses of the seed, shaken at up to half a metre a
    second."""
    nx, ny, nz = _dims(case)
    body = rigs.lattice_body_fast(np.random.default_rng(3), dims=(nx, ny, nz))
    body["node_flags"][: ny * nz] |= rigs.NF_FIXED
    rng = np.random.default_rng(seed)
    body["k"] = (body["k"] * rng.uniform(0.9, 1.1, len(body["k"]))).astype(np.float32)
    sb = SoftBody.from_arrays(body)
    free = sb.nodes["inv_mass"] > 0
    v = rng.uniform(-0.5, 0.5, sb.nodes["v"].shape).astype(np.float32)
    sb.nodes["v"] = np.where(free[:, None], v, np.float32(0))
    return sb


_LAYERS = ((64, 36), (64, 64), (64, 64), (12, 64))  # the network's weight matrices (outputs x inputs)


def _network(case, seed):
    """Weights, samples, targets and target weights as the recording step leaves them (features of order one)."""
    rng = np.random.default_rng(seed)
    parts = []
    for o, i in _LAYERS:
        parts += [rng.uniform(-1.0, 1.0, (o, i)) * math.sqrt(6.0 / i), rng.uniform(-0.05, 0.05, o)]
    p = np.concatenate([a.ravel() for a in parts]).astype(np.float32)
    n = case["samples"]
    x = rng.standard_normal((n, 36), np.float32)
    t = rng.standard_normal((n, 12), np.float32)
    w = rng.random((n, 12), np.float32)
    return p, x, t, w


def prepare(case, seed):
    kind = case["kind"]
    if kind == "substep":
        sb = _truss(case, seed)
        ptr, inc = _incidence(sb.beams, len(sb.nodes))
        dev = torch.device("cuda", 0)
        return {"kind": kind, "lib": _lib.lib(), "n": len(sb.nodes), "m": len(sb.beams),
                "nodes": torch.from_numpy(sb.nodes.copy().view(np.float32).reshape(-1, 8)).to(dev),
                "beams": torch.from_numpy(sb.beams.copy().view(np.int32).reshape(-1, 13)).to(dev),
                "ptr": torch.from_numpy(ptr).to(dev), "inc": torch.from_numpy(inc).to(dev), "g": (C.c_float * 3)(*GRAVITY)}
    if kind == "network":
        p, x, t, w = _network(case, seed)
        world = World(WorldSettings())
        world.set_mlp_weights(p)
        return {"kind": kind, "op": case["op"], "world": world, "x": x, "t": t, "w": w}
    world = world_from_rig(_rig(case, seed))
    stream = _stream()
    state = {"kind": kind, "world": world, "stream": stream, "substeps": case["substeps"]}
    if case.get("rig") == "wheeled":
        for k, wh in enumerate(rigs.wheeled_car(seed, dims=_dims(case))["bodies"][0]["wheels"]):
            if wh["propulsed"]:
                world.bodies()[0].set_wheel_drive(k, 300.0)
    for _ in range(case.get("warm", 1)):
        world.step_substeps(case["substeps"], stream)
    state["nodes"] = torch.as_tensor(_DeviceNodes(world), device="cuda")
    if "warm" in case:
        with torch.cuda.stream(stream):
            state["start"] = state["nodes"].clone()
    stream.synchronize()
    return state


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "substep":
        s = state
        rc = s["lib"].bl_gpu_substep_noalloc(s["nodes"].data_ptr(), s["n"], s["beams"].data_ptr(), s["m"], s["ptr"].data_ptr(),
                                             s["inc"].data_ptr(), C.cast(s["g"], C.c_void_p), DT, 1, 1, 0, None)
        if rc != 0:
            raise RuntimeError(f"bl_gpu_substep_noalloc: {rc}")
        # (a beam record's floats: L, k, d, max_pos, max_neg, strength, plastic, stress, L0, support_limit)
        return {"nodes": s["nodes"], "beams": s["beams"][:, 2:12].view(torch.float32)}
    if kind == "network":
        if state["op"] == "forward":
            return state["world"].mlp_forward(state["x"])
        grad, loss = state["world"].mlp_gradient(state["x"], state["t"], state["w"])
        return {"grad": grad, "loss": loss}
    stream = state["stream"]
    if "start" in state:
        with torch.cuda.stream(stream):
            state["nodes"].copy_(state["start"])
    state["world"].step_substeps(state["substeps"], stream)
    return state["nodes"]


# ------------------------------------------------------------------------------------------ what a pass cannot do without
@functools.lru_cache(maxsize=64)
def _counts(kind, key):
    case = dict(key)
    rig = rigs.shell_body(case["target"]) if kind == "shell" else _rig(dict(case, kind=kind), 1)
    n, m = rigs.rig_counts(rig)
    b = rig["bodies"][0]
    return n, m, len(b.get("fem_tris", ())), len(b.get("fem_members", ()))


def work(case):
    kind = case["kind"]
    if kind == "network":
        n = case["samples"]
        macs = sum(o * i for o, i in _LAYERS)
        if case["op"] == "forward":
            return {"bytes": 4 * n * (36 + 12), "flops": 2 * macs * n}
        # the forward, the data gradients (not of the first layer's inputs) and the weights' gradients
        return {"bytes": 4 * n * (36 + 12 + 12), "flops": 2 * n * (3 * macs - 64 * 36)}
    if kind == "substep":
        nx, ny, nz = _dims(case)
        n = nx * ny * nz
        m = sum((nx - abs(dx)) * (ny - abs(dy)) * (nz - abs(dz)) for dx in (-1, 0, 1) for dy in (-1, 0, 1) for dz in (-1, 0, 1)
                if (dx, dy, dz) > (0, 0, 0))
        m -= 2 * (nx - 1) * (ny - 1) * (nz - 1)  # (about half of the space diagonals come out longer than the rule allows)
        return {"bytes": 40 * m + 52 * n, "flops": 60 * m + 30 * n}
    steps = case["substeps"]
    n, m, tris, members = _counts(kind, tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "warm", "substeps", "kind"))))
    if kind in ("vehicle", "pair", "fleet"):
        # a beam reads its ends, L, k, d, limits and flags and writes its stress (40 B); a node is read and written
        # (52 B); once a pass where the state fits on the chip, once a substep where it does not (over 126 MB)
        per = 40 * m + 52 * n
        return {"bytes": per * (steps if per > 126e6 else 1), "flops": (60 * m + 60 * n) * steps}
    # the implicit step: a triangle's stored stiffness and rest frame (162 + 18 floats) and the frame nodes' state read
    # once (once a substep over 126 MB), the nodes written; the factorization of the minimum-degree order, 432 flops a
    # 6 x 6 block update - about 5 n^1.5 of them on a plate, growing towards 16 n^1.5 on the 50 k-node body
    per = 4 * 180 * tris + 8 * 150 * members + 120 * n
    updates = 3 * members if kind == "ladder" else n ** 1.5 * max(2.0, 2.9 * math.log(max(n, 2)) - 16.0 + (1.0 if kind == "shell" else 0.0))
    return {"bytes": per * (steps if per > 126e6 else 1) + 60 * n, "flops": steps * (432.0 * updates + 1500.0 * tris + 4000.0 * members)}


# ------------------------------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    """What run() returns for a fresh state, in float64 with numpy: the substep and the network. The worlds have none:
    a crashing frame's contacts and an implicit frame's elements restated in numpy take far too long."""
    kind = case["kind"]
    if kind == "substep":
        sb = _truss(case, seed)
        nd, bm = sb.nodes, sb.beams
        p, v, inv, mass = (np.asarray(nd[k], np.float64) for k in ("p", "v", "inv_mass", "mass"))
        a, b = bm["a"].astype(np.int64), bm["b"].astype(np.int64)
        d = p[a] - p[b]
        ln = np.sqrt((d * d).sum(1))
        stress = -bm["k"].astype(np.float64) * (ln - bm["L"]) - bm["d"].astype(np.float64) * ((v[a] - v[b]) * d).sum(1) / ln
        fv = d * (stress / ln)[:, None]
        f = mass[:, None] * np.asarray(np.asarray(GRAVITY, np.float32), np.float64)
        np.add.at(f, a, fv)
        np.add.at(f, b, -fv)
        dt = float(np.float32(DT))
        free = (inv > 0)[:, None]
        v2 = np.where(free, v + f * (inv * dt)[:, None], v)
        p2 = np.where(free, p + v2 * dt, p)
        nodes = np.concatenate([p2, inv[:, None], v2, mass[:, None]], 1)
        # (nothing yields or breaks at these speeds: the records stay as they are but for the stress)
        cols = [bm[k].astype(np.float64) for k in ("L", "k", "d", "max_pos", "max_neg", "strength", "plastic")]
        beams = np.stack(cols + [stress, bm["L0"].astype(np.float64), bm["support_limit"].astype(np.float64)], 1)
        return {"nodes": nodes, "beams": beams}
    if kind != "network":
        return None
    p, x, t, w = _network(case, seed)
    # (the network's parameters are bfloat16 values)
    p = torch.from_numpy(p)
    x, t, w = x.astype(np.float64), t.astype(np.float64), w.astype(np.float64)
    W, bias, o = [], [], 0
    for r, c in _LAYERS:
        W.append(p[o:o + r * c].to(torch.bfloat16).double().numpy().reshape(r, c))
        bias.append(p[o + r * c:o + r * c + r].to(torch.bfloat16).double().numpy())
        o += r * c + r
    h = [x]
    for k in range(4):
        z = h[-1] @ W[k].T + bias[k]
        h.append(np.maximum(z, 0.0) if k < 3 else z)
    if case["op"] == "forward":
        return h[-1]
    n = len(x)
    e = h[-1] - t
    loss = float((w * e * e).sum() / (2 * n))
    g = w * e / n
    parts = []
    for k in (3, 2, 1, 0):
        parts.append(np.concatenate([(g.T @ h[k]).ravel(), g.sum(0)]))
        if k:
            g = (g @ W[k]) * (h[k] > 0)
    return {"grad": np.concatenate(parts[::-1]), "loss": loss}
