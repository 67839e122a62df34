"""The work a user of this framework has it do, as cases that can be timed.

Scenes.  ``rollout``: the state is set from page-locked host memory, the
scene is stepped, and positions, velocities and spins are taken in sphere-id
order on the GPU (a parameter study, a data set for a learned model): every
pass starts from the same state.  ``host_loop``: the host owns the state and
exchanges it at every step (co-simulation).  ``drum`` and ``hulls``: rigid
clumps in a turning mesh and convex hulls; their bodies cannot be set, so a
pass continues where the last one ended.

Operators.  ``boxes``: the exact broad phase over boxes, by sweep and prune
or by the bounding-volume tree.  ``sort``: the radix sort of (key, value)
pairs.  ``hash``: the reference-compatible collision list, its sort and its
candidate pairs.  ``network``: training and inference of the GJK warm-start
network.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import stardust_gb300 as sd
from stardust_gb300 import _abi, scenes

FIELDS = (_abi.SD_FIELD_POSITION, _abi.SD_FIELD_VELOCITY, _abi.SD_FIELD_OMEGA)
TILE = 32_768  # spheres of one random packing; larger scenes are mirrored copies of it


def listed():
    return [
        # the plain box (4,096 equal spheres on a jittered lattice): each step is a few microseconds of work
        {"name": "box_4096", "kind": "rollout", "scene": "lattice", "n": 4096, "steps": 100},
        # the settling box: 1,048,576 polydisperse spheres falling, few contacts
        {"name": "settle_1m", "kind": "rollout", "scene": "falling", "n": 1_048_576, "steps": 40},
        # a loaded bed, a ragged count: some four contacts per sphere at every step
        {"name": "bed_199999", "kind": "rollout", "scene": "bed", "n": 199_999, "steps": 50},
        # co-simulation: state up, one step, state and contact forces down, at every step
        {"name": "host_loop_131k", "kind": "host_loop", "scene": "bed", "n": 131_072, "steps": 4},
        # independent boxes of 256 to 65,536 spheres, stepped together
        {"name": "batch_256", "kind": "rollout", "scene": "batch", "n": 256, "steps": 20},
        # a turning drum: mesh of 20,480 triangles, a tenth of the bodies 4-sphere clumps
        {"name": "drum_400k", "kind": "drum", "n": 400_000, "steps": 20},
        # convex hulls of 8 to 32 points, warm start trained online while the scene steps
        {"name": "hulls_32k", "kind": "hulls", "n": 32_768, "seed_mode": "learned", "steps": 10},
        # exact broad phase at the size of a large scene, boxes of one size
        {"name": "sap_2m", "kind": "boxes", "engine": "sap", "n": 2_000_000, "spread": 0.0},
        # the same by the tree, an ordinary size, boxes of mixed sizes
        {"name": "lbvh_300k", "kind": "boxes", "engine": "lbvh", "n": 300_001, "spread": 0.25},
        # Morton-code sized keys, a ragged count
        {"name": "sort_4m_30bit", "kind": "sort", "n": 4_000_037, "bits": 30},
        # the reference's own operator chain over 1,048,576 spheres (9 entries each)
        {"name": "hash_1m", "kind": "hash", "n": 1_048_576},
        # the warm-start network: ten Adam steps, then one forward pass
        {"name": "network_100k", "kind": "network", "n": 100_003, "iters": 10},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["rollout", "rollout", "rollout", "host_loop", "drum", "hulls", "boxes", "boxes", "sort",
                       "hash", "network"])
    if kind == "rollout":
        scene = rng.choice(["lattice", "falling", "bed", "batch"])
        n = {"lattice": lambda: rng.randint(6, 40) ** 3, "falling": lambda: _log(rng, 2_000, 1_000_000),
             "bed": lambda: _log(rng, 1_000, 300_000), "batch": lambda: _log(rng, 2, 256)}[scene]()
        return {"kind": kind, "scene": scene, "n": n, "steps": rng.randint(10, 40)}
    if kind == "host_loop":
        return {"kind": kind, "scene": rng.choice(["falling", "bed"]), "n": _log(rng, 1_000, 200_000),
                "steps": rng.randint(2, 5)}
    if kind == "drum":
        return {"kind": kind, "n": _log(rng, 4_000, 400_000), "steps": rng.randint(8, 20)}
    if kind == "hulls":
        return {"kind": kind, "n": _log(rng, 200, 32_000), "seed_mode": rng.choice(["plain", "previous", "learned"]),
                "steps": rng.randint(4, 10)}
    if kind == "boxes":
        return {"kind": kind, "engine": rng.choice(["sap", "lbvh"]), "n": _log(rng, 1_000, 2_000_000),
                "spread": rng.choice([0.0, 0.25])}
    if kind == "sort":
        return {"kind": kind, "n": _log(rng, 5_000, 9_000_000), "bits": rng.randint(10, 32)}
    if kind == "hash":
        return {"kind": kind, "n": _log(rng, 2_000, 1_000_000)}
    return {"kind": kind, "n": _log(rng, 1_000, 100_000), "iters": rng.randint(1, 10)}


# ------------------------------------------------------------------ scenes


def _falling(n, rng):
    """n polydisperse spheres at the settling box's packing, falling: one random packing, mirrored copies of it
    side by side, every copy with its own velocities."""
    m = min(n, TILE)
    box = scenes.scaled_box(m)
    pos, vel, cfg, dt, _ = scenes.settling_rsa(m, box=box, seed=int(rng.integers(1 << 31)))
    copies = -(-n // m)
    side = math.ceil((2 * copies) ** (1 / 3))  # the tile is twice as high as wide
    dims = (side, side, -(-copies // (side * side)))
    out = np.tile(pos, (copies, 1))
    for c in range(copies):
        at = np.array((c % side, c // side % side, c // (side * side)))
        part = out[c * m:(c + 1) * m]
        for a in range(3):
            if rng.integers(2):
                part[:, a] = np.float32(box[a]) - part[:, a]
            part[:, a] += np.float32(at[a] * box[a])
    v = np.empty((n, 4), np.float32)
    v[:, :3] = rng.uniform(-0.01, 0.01, (n, 3)) + (0.0, 0.0, -0.05)
    v[:, 3] = np.tile(vel[:, 3], copies)[:n]
    cfg.box_hi = tuple(float(d * b) for d, b in zip(dims, box))
    return out[:n], v, cfg, dt


def _bed(n, rng):
    """n nearly equal spheres in a loaded body-centred packing on the floor of a box, some four of each sphere's
    eight neighbours in contact."""
    r = 0.005
    a = 4.0 * r / math.sqrt(3.0)
    k = max(2, round((n / 2) ** (1 / 3)))
    layers = -(-n // (2 * k * k))
    g = np.stack(np.meshgrid(np.arange(layers), np.arange(k), np.arange(k), indexing="ij"), -1).reshape(-1, 3)[:, ::-1]
    pos = np.empty((2 * len(g), 4), np.float32)
    pos[0::2, :3] = g * a + r
    pos[1::2, :3] = (g + 0.5) * a + r
    pos = pos[:n]
    pos[:, :3] += rng.uniform(-0.001 * r, 0.001 * r, (n, 3))
    pos[:, 3] = r * rng.uniform(0.9985, 1.0025, n)
    vel = np.empty((n, 4), np.float32)
    vel[:, :3] = rng.uniform(-0.005, 0.005, (n, 3))
    vel[:, 3] = scenes.DENSITY * 4.0 / 3.0 * math.pi * pos[:, 3].astype(np.float64) ** 3
    edge = (k - 0.5) * a + 2 * r
    cfg = sd.EngineConfig(box_hi=(edge, edge, 1.5 * layers * a + 2 * r), cell=2.01 * r, pair_capacity=1 << 22)
    return pos, vel, cfg, 5e-6


def _batch_counts(n):
    """Sphere counts of n scenes, lognormal about 4,096 in [256, 65,536]; the same for every seed."""
    z = np.random.default_rng(n).normal(size=n)
    return np.clip(np.round(4096 * np.exp(0.85 * z)), 256, 65_536).astype(int)


def _batch(n, rng):
    """n independent boxes of equal spheres on jittered lattices, at 35 % of their volume."""
    r = scenes.R_BOX
    gap = r * (4.0 / 3.0 * math.pi / 0.35) ** (1 / 3)
    pos, vel, spans, first = [], [], [], 0
    for k in _batch_counts(n):
        side = math.ceil(round(float(k) ** (1 / 3), 6))
        p, v = sd.scene_lattice(side, side, side, gap, 0.05 * r, (0.5 * gap,) * 3, r, scenes.M_BOX, 0.1,
                                int(rng.integers(1 << 31)))
        pos.append(p[:k])
        vel.append(v[:k])
        spans.append((first, first + int(k), (0.0, 0.0, 0.0), (side * gap,) * 3))
        first += int(k)
    return np.concatenate(pos), np.concatenate(vel), sd.EngineConfig(pair_capacity=1 << 22), 1e-5, spans


def _spheres(case, seed):
    """(positions, velocities, spins, config, dt, scenes): scenes is a list of (first, last, lo, hi)."""
    rng = np.random.default_rng(seed)
    n, spans = case["n"], None
    if case["scene"] == "batch":
        pos, vel, cfg, dt, spans = _batch(n, rng)
    elif case["scene"] == "lattice":
        side = round(n ** (1 / 3))
        pos, vel, cfg, dt = scenes.box_lattice(side, seed=int(rng.integers(1 << 31)))
        edge = (side + 14) * 2.2 * scenes.R_BOX  # room around the lattice, as in the 4,096-sphere box
        pos[:, :3] += np.float32((edge - 0.64) / 2.0)
        cfg.box_hi = (edge, edge, edge)
    elif case["scene"] == "falling":
        pos, vel, cfg, dt = _falling(n, rng)
    else:
        pos, vel, cfg, dt = _bed(n, rng)
    omg = np.zeros_like(pos)
    omg[:, :3] = rng.uniform(-2.0, 2.0, (len(pos), 3))
    return pos, vel, omg, cfg, dt, spans or [(0, len(pos), cfg.box_lo, cfg.box_hi)]


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).pin_memory()


def _sphere_engine(case, seed):
    pos, vel, omg, cfg, dt, spans = _spheres(case, seed)
    if case["kind"] == "host_loop":
        cfg.flags = _abi.SD_FLAG_RECORD
    eng = sd.DEMEngine(cfg)
    if case["scene"] == "batch":
        for a, b, lo, hi in spans:
            eng.add_scene(pos[a:b], vel[a:b], lo, hi)
    else:
        eng.add_spheres(pos, vel)
    eng.prepare()
    start = [_pinned(x) for x in (pos, vel, omg)]
    return {"eng": eng, "dt": dt, "start": start}


class _Device:
    """A float4 field of the engine (or, with ids, the sphere ids of its slots) as torch sees it; keeps the engine."""

    def __init__(self, eng, field):
        self.eng = eng
        ids = field == _abi.SD_FIELD_IDS
        self.__cuda_array_interface__ = {
            "data": (eng.device_ptr(field), False), "version": 3, "typestr": "<i4" if ids else "<f4",
            "shape": (eng.n,) if ids else (eng.n, 4), "strides": (16,) if ids else None}


def _by_id(eng):
    """Positions, velocities and spins in sphere-id order, on the GPU."""
    stream = torch.cuda.ExternalStream(eng.stream())
    with torch.cuda.stream(stream):
        ids = torch.as_tensor(_Device(eng, _abi.SD_FIELD_IDS), device="cuda").long() & 0x7FFFFFFF
        out = []
        for f in FIELDS:
            src = torch.as_tensor(_Device(eng, f), device="cuda")
            dst = torch.empty((eng.n, 3), dtype=torch.float32, device="cuda")
            dst[ids] = src[:, :3]
            out.append(dst)
    eng.sync()  # waits for the steps and raises what the device reports
    return dict(zip(("pos", "vel", "omg"), out))


def _run_rollout(s):
    eng = s["eng"]
    for f, host in zip(FIELDS, s["start"]):
        eng.set(f, host.numpy())
    eng.step(s["dt"], s["steps"])
    return _by_id(eng)


def _transfer(name, eng, field, host):
    _abi.call(name, eng._h, field, ctypes.c_void_p(host.data_ptr()), host.numel() * 4, h=eng._h)


def _run_host_loop(s):
    eng, (pos, vel, force) = s["eng"], s["host"]
    pos.copy_(s["start"][0])
    vel.copy_(s["start"][1])
    _transfer("sd_engine_set_state", eng, _abi.SD_FIELD_OMEGA, s["start"][2])
    for _ in range(s["steps"]):
        _transfer("sd_engine_set_state", eng, _abi.SD_FIELD_POSITION, pos)
        _transfer("sd_engine_set_state", eng, _abi.SD_FIELD_VELOCITY, vel)
        eng.step(s["dt"], 1)
        _transfer("sd_engine_get_state", eng, _abi.SD_FIELD_POSITION, pos)
        _transfer("sd_engine_get_state", eng, _abi.SD_FIELD_VELOCITY, vel)
        _transfer("sd_engine_get_state", eng, _abi.SD_FIELD_FORCE, force)
    return {"pos": pos[:, :3], "vel": vel[:, :3], "force": force[:, :3]}


def _drum_engine(case, seed):
    """The rotating drum of scenes.drum_scene, built with array operations; the drum keeps its length and its mesh,
    and holds the bodies that n asks for."""
    rng = np.random.default_rng(seed)
    n, radius, length, rmin, rmax, density = case["n"], 0.5, 0.5, 0.0012, 0.0024, 2500.0
    grow = max(1.0, (1_000_000 / n) ** (1 / 3))  # fewer spheres are larger ones: the drum is as full
    rmin, rmax = rmin * grow, rmax * grow
    tris, patch = scenes.drum_mesh(radius, length, 128, 65, 8, (0.5 * length, radius, radius))
    sp, margin = 2.1 * rmax, 1.2 * rmax
    xs = np.arange(margin, length - margin, sp)
    ys = np.arange(margin, 2 * radius - margin, sp)
    sites = np.stack(np.meshgrid(ys, ys, xs, indexing="ij"), -1).reshape(-1, 3)[:, ::-1]  # (x, y, z), lowest z first
    sites = sites[(sites[:, 1] - radius) ** 2 + (sites[:, 2] - radius) ** 2 < (radius - margin) ** 2]
    bodies = min(len(sites), int(n / 1.3))
    sites = sites[:bodies] + rng.uniform(-0.02 * rmax, 0.02 * rmax, (bodies, 3))
    is_clump = rng.permutation(bodies) < bodies // 10
    cfg = sd.EngineConfig(box_hi=(length, 2 * radius, 2 * radius), walls=0, cell=2 * rmax, pair_capacity=1 << 22)
    eng = sd.DEMEngine(cfg)
    tet = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]]) * (0.6 / math.sqrt(3.0))
    for com, r in zip(sites[is_clump], rng.uniform(rmin, 0.75 * rmax, int(is_clump.sum()))):
        rel = np.concatenate([tet * r, np.full((4, 1), r)], 1).astype(np.float32)
        eng.add_clump(rel, density * 16.0 / 3.0 * math.pi * r ** 3, tuple(com), (0.0, 0.0, -0.1))
    free = sites[~is_clump]
    r = rng.uniform(rmin, rmax, len(free))
    pos = np.concatenate([free, r[:, None]], 1).astype(np.float32)
    vel = np.zeros_like(pos)
    vel[:, 2] = -0.1
    vel[:, 3] = density * 4.0 / 3.0 * math.pi * r ** 3
    eng.add_spheres(pos, vel)
    eng.add_mesh(tris, (0.5 * length, radius, radius), (1.0, 0.0, 0.0), 2.0, patch)
    eng.prepare()
    return {"eng": eng, "dt": 2e-6}


def _run_drum(s):
    s["eng"].step(s["dt"], s["steps"])
    return _by_id(s["eng"])


def _hull_engine(case, seed):
    n = case["n"]
    edge = max(0.2, 0.02 * (3 + math.ceil((2 * n) ** (1 / 3))))
    pts, pos, quat, vel, mass, cfg, dt = scenes.hull_box(n, seed=seed, box=(edge,) * 3, spacing=0.02, vmax=0.2)
    eng = sd.DEMEngine(cfg)
    sd.add_hull_scene(eng, pts, pos, quat, vel, mass)
    eng.prepare()
    mode = {"plain": _abi.SD_GJK_SEED_PLAIN, "previous": _abi.SD_GJK_SEED_PREVIOUS,
            "learned": _abi.SD_GJK_SEED_LEARNED}[case["seed_mode"]]
    eng.set_gjk_seed(mode)
    if case["seed_mode"] == "learned":
        eng.set_gjk_training(5, 10, 2e-3)
    return {"eng": eng, "dt": dt, "host": [torch.empty((n, 4), pin_memory=True) for _ in range(3)]}


def _run_hulls(s):
    eng, out = s["eng"], {}
    eng.step(s["dt"], s["steps"])
    for name, f, host in zip(("pos", "vel", "quat"), (_abi.SD_BODY_POSITION, _abi.SD_BODY_VELOCITY,
                                                       _abi.SD_BODY_QUATERNION), s["host"]):
        _transfer("sd_engine_get_bodies", eng, f, host)
        out[name] = host if name == "quat" else host[:, :3]
    return out


# --------------------------------------------------------------- operators


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _boxes(case, seed):
    """Boxes uniform in the unit cube, about 4 overlaps each whatever their number; spread: half-widths lognormal."""
    g, n = _generator(seed), case["n"]
    c = torch.rand((n, 3), generator=g, device="cuda")
    size = torch.exp(case["spread"] * torch.randn((n, 3), generator=g, device="cuda") - 0.75 * case["spread"] ** 2)
    half = 0.5 * (0.5 / n) ** (1 / 3) * size
    lo, hi = torch.zeros((n, 4), device="cuda"), torch.zeros((n, 4), device="cuda")
    lo[:, :3], hi[:, :3] = c - half, c + half
    cap = 4 * n
    op = sd.SweepAndPrune if case["engine"] == "sap" else sd.BoundingVolumes
    return {"entry": f"sd_{case['engine']}_pairs", "n": n, "lo": lo, "hi": hi, "cap": cap,
            "pairs": torch.zeros(cap, dtype=torch.int64, device="cuda"),
            "count": torch.zeros(2, dtype=torch.int32, device="cuda"),
            "scratch": torch.empty(op.scratch_bytes(n, cap), dtype=torch.uint8, device="cuda")}


def _run_boxes(s):
    """The operator as a program with its own buffers calls it: ascending pairs, their number and the error bits."""
    _abi.call(s["entry"], s["n"], s["lo"].data_ptr(), s["hi"].data_ptr(), s["pairs"].data_ptr(), s["cap"],
              s["count"].data_ptr(), s["scratch"].data_ptr(), s["scratch"].numel(),
              torch.cuda.current_stream().cuda_stream)
    return {"pairs": s["pairs"], "count": s["count"]}


def _sort(case, seed):
    g, n, bits = _generator(seed), case["n"], case["bits"]
    keys = torch.randint(0, 1 << bits, (n,), generator=g, device="cuda").to(torch.int32)
    scratch = torch.zeros(sd.SpatialPartition.sort_scratch_bytes(n, bits), dtype=torch.uint8, device="cuda")
    return {"n": n, "bits": bits, "src": keys, "ids": torch.arange(n, dtype=torch.int32, device="cuda"),
            "buf": [torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(4)], "scratch": scratch}


def _run_sort(s):
    keys, vals, keys_tmp, vals_tmp = s["buf"]
    keys.copy_(s["src"])
    vals.copy_(s["ids"])
    sd.SpatialPartition.sort_pairs(keys, vals, keys_tmp, vals_tmp, s["n"], s["bits"], s["scratch"])
    return {"keys": keys, "vals": vals}


def _hash(case, seed):
    """Spheres in the unit cube, one per cell on average (at most 255 cells per axis)."""
    g, n = _generator(seed), case["n"]
    per_axis = min(250, max(4, round(n ** (1 / 3))))
    cell = 1.0 / per_axis
    pos = torch.rand((n, 4), generator=g, device="cuda")
    size = cell * (0.2 + 0.2 * torch.rand(n, generator=g, device="cuda"))
    entries, cap = 9 * n, 12 * n
    new = lambda k, t: torch.zeros(k, dtype=t, device="cuda")  # noqa: E731
    return {"n": n, "cell": cell, "pos": pos, "size": size, "cap": cap,
            "buf": [new(entries, torch.int32) for _ in range(4)], "count": new(1, torch.int32),
            "sort_scratch": new(sd.SpatialPartition.sort_scratch_bytes(entries), torch.uint8),
            "pair_scratch": new(sd.SpatialPartition.pairs_scratch_bytes(entries), torch.uint8),
            "pairs": [new(cap, torch.int32) for _ in range(2)], "npairs": new(1, torch.int64)}


def _run_hash(s):
    P, n = sd.SpatialPartition, s["n"]
    cells, ids, cells_tmp, ids_tmp = s["buf"]
    P.construct_collision_list(n, s["cell"], cells, ids, s["size"], s["pos"], s["count"])
    P.sort_collision_list(cells, ids, cells_tmp, ids_tmp, 9 * n, s["sort_scratch"])
    P.candidate_pairs(cells, ids, s["count"], 9 * n, None, *s["pairs"], s["cap"], s["npairs"], s["pair_scratch"])
    return {"cells": cells, "ids": ids, "a": s["pairs"][0], "b": s["pairs"][1], "npairs": s["npairs"]}


def _network_inputs(case, seed):
    """Inputs as hull scenes give them (relative quaternion, centre offset, flag, previous direction, distance) and
    targets a few degrees off the previous direction; the initial parameters of a training run."""
    rng, n = np.random.default_rng(seed), case["n"]
    unit = lambda a: a / np.linalg.norm(a, axis=1, keepdims=True)  # noqa: E731
    feat = np.zeros((n, 16), np.float32)
    feat[:, :4] = unit(rng.normal(size=(n, 4)))
    feat[:, 4:7] = unit(rng.normal(size=(n, 3))) * rng.uniform(0.6, 1.0, (n, 1))
    feat[:, 7] = 1.0
    feat[:, 8:11] = unit(feat[:, 4:7] + 0.3 * rng.normal(size=(n, 3)))
    feat[:, 11] = np.linalg.norm(feat[:, 4:7], axis=1)
    target = np.ones((n, 4), np.float32)
    target[:, :3] = unit(feat[:, 8:11] + 0.15 * rng.normal(size=(n, 3)))
    w = rng.uniform(-1.0, 1.0, 6288).astype(np.float32)
    w[:1024] /= 4.0
    w[1024:1088] = 0.0
    w[1088:5184] /= 8.0
    w[5184:5248] = 0.0
    w[5248:5248 + 192] /= 16.0
    w[5248 + 192:] = 0.0
    return feat, target, w


def _network(case, seed):
    feat, target, w = _network_inputs(case, seed)
    eng = sd.DEMEngine(sd.EngineConfig())
    cube = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], np.float32) * 0.01
    for k in range(2):
        eng.add_hull(cube, 1e-3, (0.3 + 0.1 * k, 0.5, 0.5))
    eng.prepare()
    return {"eng": eng, "feat": torch.from_numpy(feat).cuda(), "target": torch.from_numpy(target).cuda(), "w": w,
            "iters": case["iters"]}


def _run_network(s):
    eng = s["eng"]
    eng.set_mlp_params(s["w"])
    grad = eng.mlp_train(s["feat"], s["target"], s["iters"], 1e-3)
    return {"grad": grad, "params": eng.mlp_params(), "out": eng.mlp_forward(s["feat"])[:, :3]}


# ---------------------------------------------------------------- contract

_PREPARE = {"rollout": _sphere_engine, "host_loop": _sphere_engine, "drum": _drum_engine, "hulls": _hull_engine,
            "boxes": _boxes, "sort": _sort, "hash": _hash, "network": _network}
_RUN = {"rollout": _run_rollout, "host_loop": _run_host_loop, "drum": _run_drum, "hulls": _run_hulls,
        "boxes": _run_boxes, "sort": _run_sort, "hash": _run_hash, "network": _run_network}


def prepare(case, seed):
    torch.cuda.init()
    s = _PREPARE[case["kind"]](case, seed)
    s["kind"], s["steps"] = case["kind"], case.get("steps", 1)
    if case["kind"] == "host_loop":
        s["host"] = [torch.empty_like(s["start"][0], pin_memory=True) for _ in range(3)]
    return s


def run(state):
    return _RUN[state["kind"]](state)


def work(case):
    """A step reads and writes each sphere's or body's state once (a hull also its vertices, 20 on average); an
    operator reads its inputs and writes its results once."""
    kind, n, steps = case["kind"], case["n"], case.get("steps", 1)
    if kind in ("rollout", "host_loop", "drum"):
        if case.get("scene") == "batch":
            n = int(_batch_counts(n).sum())
        if case.get("scene") == "lattice":
            n = round(n ** (1 / 3)) ** 3
        state, flops = 96.0 * n, 60.0 * n
        if case.get("scene") == "bed":
            flops += 4 * 150.0 * n
        if kind == "host_loop":
            state += 80.0 * n  # up and down the host link, and the forces
        return {"bytes": state * steps, "flops": flops * steps}
    if kind == "hulls":
        return {"bytes": (2 * 80.0 + 16 * 20 + 3 * 8) * n * steps, "flops": 3 * 3 * 40 * 5.0 * n * steps}
    if kind == "boxes":
        return {"bytes": 32.0 * n + 2.0 * n * 8, "flops": 6.0 * n}
    if kind == "sort":
        return {"bytes": 16.0 * n, "flops": 0.0}
    if kind == "hash":
        return {"bytes": (20.0 + 2 * 9 * 8) * n, "flops": 60.0 * n}
    gemm = 2.0 * (16 * 64 + 64 * 64 + 64 * 16)
    return {"bytes": (80.0 * case["iters"] + 64 + 16) * n, "flops": gemm * n * (3 * case["iters"] + 1)}


# ----------------------------------------------------------------- 64 bits


def _neighbours(x, cell, scene):
    """(i, j), each unordered pair once: spheres of one scene in the same or adjacent cells of the given edge."""
    c = ((x - x.min(0).values) / cell).long() + 1
    dims = c.max(0).values + 2
    key = ((scene * dims[0] + c[:, 0]) * dims[1] + c[:, 1]) * dims[2] + c[:, 2]
    key, order = key.sort()
    at = torch.arange(len(key), device=x.device)
    for step in range(14):  # half of the 27 offsets, the own cell last
        d = (1, step % 3 - 1, step // 3 - 1) if step < 9 else (0, 1, step - 10) if step < 12 else (0, 0, 13 - step)
        other = key + (d[0] * dims[1] + d[1]) * dims[2] + d[2]
        first = at + 1 if step == 13 else torch.searchsorted(key, other)
        count = torch.searchsorted(key, other, right=True) - first
        i = torch.repeat_interleave(at, count)
        k = torch.arange(len(i), device=x.device) - torch.repeat_interleave(count.cumsum(0) - count, count)
        yield order[i], order[torch.repeat_interleave(first, count) + k]


def _response(cfg, n, delta, dv, ws, meff, r):
    """The spring-dashpot law: force on the sphere that n points to, and n x (tangential force)."""
    le = math.log(cfg.restitution)
    gamma = 2.0 * -le / math.sqrt(math.pi ** 2 + le * le) * math.sqrt(cfg.kn) * meff.sqrt()[:, None]
    v = dv - torch.linalg.cross(ws, n)
    vn = (v * n).sum(1, keepdim=True)
    fn = cfg.kn * delta[:, None] - gamma * vn
    vt = v - vn * n
    speed = vt.norm(dim=1, keepdim=True)
    ft = -torch.minimum(cfg.mu * fn.clamp(min=0), gamma * speed) * vt / speed.clamp(min=1e-300)
    return fn * n + ft, torch.linalg.cross(n, ft)


def _exact_spheres(case, seed):
    pos, vel, omg, cfg, dt, spans = _spheres(case, seed)
    x, v, w = (torch.from_numpy(a[:, :3]).double().cuda() for a in (pos, vel, omg))
    r, m = (torch.from_numpy(np.ascontiguousarray(a[:, 3])).double().cuda() for a in (pos, vel))
    lo, hi = torch.empty_like(x), torch.empty_like(x)
    scene = torch.empty(len(x), dtype=torch.long, device="cuda")
    for k, (a, b, l, h) in enumerate(spans):
        lo[a:b], hi[a:b] = (torch.tensor(np.float32(q), device="cuda").double() for q in (l, h))
        scene[a:b] = k
    f = torch.zeros_like(x)
    g = torch.tensor(np.float32(cfg.gravity), device="cuda").double()
    dt = float(np.float32(dt))
    reach = 2.0 * case["steps"] * dt * (1.0 + float(v.norm(dim=1).max()))  # no pair closes in by more
    near = []
    for i, j in _neighbours(x, 2.0 * float(r.max()) + reach, scene):
        close = (x[i] - x[j]).norm(dim=1) < r[i] + r[j] + reach
        near.append((i[close], j[close]))
    ni, nj = (torch.cat([p[k] for p in near]) for k in (0, 1))
    for _ in range(case["steps"]):
        f, t = torch.zeros_like(x), torch.zeros_like(x)
        d = x[ni] - x[nj]
        dist = d.norm(dim=1)
        hit = dist < r[ni] + r[nj]
        i, j, d, dist = ni[hit], nj[hit], d[hit], dist[hit]
        fij, q = _response(cfg, d / dist[:, None], r[i] + r[j] - dist, v[i] - v[j], r[i, None] * w[i] + r[j, None] * w[j],
                           m[i] * m[j] / (m[i] + m[j]), r[i])
        f.index_add_(0, i, fij)
        f.index_add_(0, j, -fij)
        t.index_add_(0, i, -r[i, None] * q)
        t.index_add_(0, j, -r[j, None] * q)
        for a in range(3):
            for gap, sign in ((x[:, a] - lo[:, a], 1.0), (hi[:, a] - x[:, a], -1.0)):
                i = (gap < r).nonzero()[:, 0]
                n = torch.zeros((len(i), 3), dtype=x.dtype, device="cuda")
                n[:, a] = sign
                fw, q = _response(cfg, n, (r - gap)[i], v[i], r[i, None] * w[i], m[i], r[i])
                f.index_add_(0, i, fw)
                t.index_add_(0, i, -r[i, None] * q)
        v = v + dt * (f / m[:, None] + g)
        x = x + dt * v
        w = w + dt * t / (0.4 * m * r * r)[:, None]
    return {"pos": x, "vel": v, "force": f} if case["kind"] == "host_loop" else {"pos": x, "vel": v, "omg": w}


def _exact_network(case, seed):
    feat, target, w = (torch.from_numpy(a).double().cuda() for a in _network_inputs(case, seed))
    shapes = ((64, 16), (64,), (64, 64), (64,), (16, 64), (16,))
    w = w.clone().requires_grad_(True)

    def forward():
        p = [q.reshape(s) for q, s in zip(w.split([math.prod(s) for s in shapes]), shapes)]
        h = torch.relu(feat @ p[0].T + p[1])
        h = torch.relu(h @ p[2].T + p[3])
        return (h @ p[4].T + p[5])[:, :3] + feat[:, 8:11]

    m1, m2, grad = torch.zeros_like(w), torch.zeros_like(w), None
    for k in range(1, case["iters"] + 1):
        y = forward()
        cosine = (y * target[:, :3]).sum(1) / (y.square().sum(1) + 1e-8).sqrt()
        grad, = torch.autograd.grad((1.0 - cosine).mean(), w)
        m1, m2 = 0.9 * m1 + 0.1 * grad, 0.999 * m2 + 0.001 * grad * grad
        with torch.no_grad():
            w -= 1e-3 * (m1 / (1 - 0.9 ** k)) / ((m2 / (1 - 0.999 ** k)).sqrt() + 1e-8)
    return {"grad": grad, "params": w.detach(), "out": forward().detach()}


def exact(case, seed):
    """Sphere scenes and the network in 64 bits.  The box, sort and hash operators return whole numbers.  The drum
    (each sphere against 20,480 triangles) and the hulls (a separating-axis search over every vertex, edge and face
    of each pair) have no plain restatement that ends in seconds; they are held to their float type."""
    if case["kind"] in ("rollout", "host_loop"):
        return _exact_spheres(case, seed)
    return _exact_network(case, seed) if case["kind"] == "network" else None
