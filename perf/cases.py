"""Workloads of the TSDF integrate path, as programs that map rooms run them.

A case is one pass of such a program through the package's public entry
points, on depth frames of the seeded synthetic rooms of ``scenes`` (a 6x6x3 m
room, three spheres, two boxes, a circular camera orbit, depth noise, 5 % of
the pixels invalid), made on the GPU here. Kinds:

  session  reset, then every frame of a trajectory, ``per_call`` frames a call
           (``integrate`` or ``integrate_frames``; ``source`` "depth": the depth
           images themselves through ``integrate_depth[_frames]``; "split": the
           two stages ``allocate_blocks`` and ``update_voxels`` one by one)
  live     the same calls on a map that is kept (no reset): ``laps`` passes
           over the same frames were made before
  batch    ``scenes`` volumes of different voxel sizes and resolutions, reset,
           then one frame of each per batch step
  extract  the mesh of an integrated room, left in device buffers

``voxel`` is in metres, ``trunc`` in voxels, ``cap`` the weight cap (0: none),
``radius`` the far cutoff in metres (0: none).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from what_irregularity_costs_b200 import (STORAGE_FP16_U16, STORAGE_FP32, Batch, CudaVolume,
                                          device_tensor, scenes)

STORAGE = {"fp32": STORAGE_FP32, "fp16": STORAGE_FP16_U16}
BATCH_SIZES = [(160, 120), (320, 240), (640, 480), (1280, 720)]
MESH_VERTS = 12_000_000  # room for the mesh of a whole room at 2 cm


def _session(name, width, height, frames, per_call, **kw):
    case = {"name": name, "kind": "session", "source": "points", "width": width, "height": height,
            "frames": frames, "per_call": per_call, "voxel": 0.02, "trunc": 4.0, "cap": 64.0, "radius": 0.0,
            "storage": "fp32", "pipelined": False, "pool": 1 << 16, "laps": 0}
    case.update(kw)
    return case


def listed():
    return [
        # The smallest call: one small frame into a kept map, as a tracker on a
        # robot does per camera frame. Latency and launches count.
        _session("live small frame", 160, 120, 1, 1, kind="live", voxel=0.04, cap=0.0, pool=1 << 13, laps=1),
        # A camera that stays in a room already mapped: most voxels at the cap.
        _session("live mapped room", 640, 480, 4, 4, kind="live", laps=80),
        # Live mapping at 640x480, one call per frame: the reference's call pattern, fused.
        _session("frames one by one", 640, 480, 20, 1),
        # The benchmark's step: a whole trajectory, four frames per call, its own pool.
        _session("room trajectory", 640, 480, 100, 4, pool=1 << 19),
        # A small camera, compact storage, updates overlapping the next call's walk.
        _session("small camera fp16", 320, 240, 32, 1, storage="fp16", pipelined=True, pool=1 << 15),
        # Depth images straight from the sensor, unprojected on the GPU.
        _session("depth images", 640, 480, 16, 4, source="depth"),
        # The reference's two stages called one after the other (its own test does).
        _session("two stages", 640, 480, 8, 1, source="split"),
        # A fine map of large frames: many blocks, a large pool.
        _session("fine large frames", 1280, 720, 4, 4, voxel=0.01, pool=1 << 18),
        # Odd sizes: ragged frames, a wide band (several chunks a ray), a far cutoff, a low cap.
        _session("odd wide band", 421, 317, 7, 3, voxel=0.0171, trunc=6.5, cap=7.0, radius=3.7, pool=1 << 17),
        # Many rooms at once: mixed voxel sizes and resolutions, one frame each per step.
        {"name": "batch of scenes", "kind": "batch", "scenes": 12, "frames": 6, "storage": "fp16", "cap": 64.0,
         "shift": 0},
        # The mesh of a whole room.
        _session("mesh of a room", 640, 480, 25, 5, kind="extract", rgb=False),
        # A coloured mesh of part of a room, compact storage.
        _session("coloured mesh", 320, 240, 5, 5, kind="extract", rgb=True, voxel=0.03, storage="fp16",
                 pool=1 << 14),
    ]


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["session"] * 5 + ["live"] * 2 + ["extract", "batch"])
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(3, 14), "frames": rng.randint(3, 8),
                "storage": rng.choice(["fp16", "fp32"]), "cap": rng.choice([64.0, 16.0, 0.0]),
                "shift": rng.randint(0, 11)}
    width = int(round(math.exp(rng.uniform(math.log(120), math.log(1280)))))
    height = max(64, int(round(width * rng.uniform(0.5, 0.8))))
    voxel = round(math.exp(rng.uniform(math.log(0.01), math.log(0.04))), 5)
    trunc = rng.choice([4.0, 4.0, 4.0, 3.0, round(rng.uniform(2.0, 8.0), 2)])
    most = max(1, int(9_000_000 / (width * height * trunc / 4.0)))
    frames = min(rng.randint(1, 40), most)
    per_call = min(rng.choice([1, 1, 2, 3, 4, 8]), frames)
    # A full room has about 15 thousand blocks at 2 cm and 4 voxels of truncation.
    pool = 1 << max(12, math.ceil(math.log2(30_000 * (0.02 / voxel) ** 2 * max(1.0, trunc / 4.0))))
    case = _session("", width, height, frames, per_call, kind=kind, voxel=voxel, trunc=trunc, pool=pool,
                    cap=rng.choice([64.0, 64.0, 32.0, 6.0, 0.0]), radius=rng.choice([0.0, 0.0, 4.0]),
                    storage=rng.choice(["fp32", "fp32", "fp16"]))
    del case["name"]
    if kind == "session":
        case["source"] = rng.choice(["points", "points", "depth", "split"])
        case["pipelined"] = rng.random() < 0.2
    elif kind == "live":
        case["frames"] = case["per_call"] = min(frames, rng.choice([1, 1, 2, 4]))
        case["laps"] = rng.choice([1, 3, 70])
    else:
        case["voxel"] = max(voxel, 0.02)
        case["rgb"] = rng.random() < 0.4
    if case["source"] == "depth":
        case["radius"] = 0.0
    if case["source"] == "split":
        case["per_call"] = 1
    return case


# ---- inputs ----------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _raycast(scene, o, d):
    """Distance along the rays d (h, w, 3) from o, in units of d, to the room's
    walls, spheres and boxes."""
    inf = torch.full(d.shape[:-1], math.inf, dtype=d.dtype, device=d.device)
    vec = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=d.device)  # noqa: E731
    o = vec(o)
    inv = 1.0 / d
    hi, lo = (vec(scene.hi) - o) * inv, (vec(scene.lo) - o) * inv
    t = torch.where(d > 0, hi, torch.where(d < 0, lo, inf[..., None])).amin(-1)
    for c, r in scene.spheres:
        oc = vec(c) - o
        a, b = (d * d).sum(-1), d @ oc
        disc = b * b - a * (oc @ oc - r * r)
        near = (b - disc.clamp_min(0.0).sqrt()) / a
        t = torch.minimum(t, torch.where((disc >= 0) & (near > 1e-9), near, inf))
    for blo, bhi in scene.boxes:
        t1, t2 = (vec(blo) - o) * inv, (vec(bhi) - o) * inv
        tmin, tmax = torch.minimum(t1, t2).amax(-1), torch.maximum(t1, t2).amin(-1)
        t = torch.minimum(t, torch.where((tmax >= tmin.clamp_min(0.0)) & (tmin > 1e-9), tmin, inf))
    return t


def _frames(seed, width, height, n):
    """n orbit frames of the room of this seed: depth images (n, h, w) float32,
    rotations, camera origins and intrinsics."""
    dev = _device()
    K = scenes.ROOM_K.scaled(width, height)
    scene = scenes.RoomScene.make(seed)
    gen = torch.Generator(device=dev).manual_seed(seed)
    u = (torch.arange(width, dtype=torch.float64, device=dev) - K.cx) / K.fx
    v = (torch.arange(height, dtype=torch.float64, device=dev) - K.cy) / K.fy
    cam = torch.stack([u.expand(height, width), v[:, None].expand(height, width),
                       torch.ones(height, width, dtype=torch.float64, device=dev)], -1)
    depth = torch.empty((n, height, width), dtype=torch.float32, device=dev)
    Rs, ts = [], []
    for k in range(n):
        R, t = scenes.orbit_pose(k, np.random.default_rng([seed, k + 1]))
        z = _raycast(scene, t, cam @ torch.as_tensor(R.T.copy(), device=dev))
        z = z + torch.randn(z.shape, generator=gen, dtype=torch.float64, device=dev) * (0.0015 * z * z)
        z = torch.where(torch.rand(z.shape, generator=gen, device=dev) < 0.05, torch.zeros_like(z), z)
        depth[k] = torch.where((z >= 0.1) & (z <= 8.0), z, torch.zeros_like(z)).float()
        Rs.append(R)
        ts.append(t)
    return depth, np.stack(Rs), np.stack(ts), K


def _points(depth, R, t, K):
    """World points (n, 3) float32 of one image's valid pixels, in raster order."""
    v, u = torch.nonzero(depth > 0, as_tuple=True)
    z = depth[v, u].double()
    x = (u.double() - K.cx) * z / torch.full_like(z, K.fx)
    y = (v.double() - K.cy) * z / torch.full_like(z, K.fy)
    return torch.stack([((R[i, 0] * x + R[i, 1] * y) + R[i, 2] * z) + t[i] for i in range(3)], -1).float()


def _clouds(seed, width, height, n):
    depth, Rs, ts, K = _frames(seed, width, height, n)
    return [_points(depth[k], Rs[k], ts[k], K) for k in range(n)], ts.astype(np.float32)


def _scene_sizes(case):
    """(width, height, voxel, pool) of every scene of a batch."""
    out = []
    for i in range(case["scenes"]):
        k = i + case["shift"]
        w, h = BATCH_SIZES[(k * 7 + k // 4) % 4]
        voxel = round(0.01 * 4.0 ** ((k * 5 % 11) / 10.0), 5)
        out.append((w, h, voxel, 1 << max(12, math.ceil(math.log2(24_000 * (0.02 / voxel) ** 2)))))
    return out


# ---- outputs ---------------------------------------------------------------

def _rows(voxel, trunc, pool):
    """Rows a map is read out in: more than a whole room of these voxels fills."""
    return min(pool, int(22_000 * (0.02 / voxel) ** 2 * max(1.0, trunc / 4.0)))


def _padded(rows, n):
    """The first n of n rows and zeros."""
    if rows.shape[0] > n:
        raise RuntimeError(f"{rows.shape[0]} rows, room for {n}")
    return torch.cat([rows, rows.new_zeros((n - rows.shape[0],) + tuple(rows.shape[1:]))])


class _Blocks(dict):
    """A volume's contents, read when they are looked at: blocks by ascending
    coordinate (their order in the pool is the order of insertion, which no two
    runs share), then every voxel array, one row per block; zeros past the last."""

    def __init__(self, vol, owner, rows):
        self.vol, self.owner, self.rows, self.read = vol, owner, rows, None
        names = ["blocks", "coords", "dropped", "tsdf", "weight"] + ["r", "g", "b"] * (vol.storage == STORAGE_FP32)
        super().__init__((n, None) for n in names)

    def __getitem__(self, name):
        if self.read is None:
            torch.cuda.synchronize()
            vol, view = self.vol, self.vol.device_view()
            n = vol.block_count()
            coords = device_tensor(view.block_coord, (n, 3), "<i4").long()
            order = torch.argsort((((coords[:, 0] << 20) + coords[:, 1]) << 20) + coords[:, 2])
            half = vol.storage == STORAGE_FP16_U16
            self.read = {"blocks": n, "coords": _padded(coords[order].int(), self.rows), "dropped": vol.drop_count()}
            for key in self:
                if key in self.read:
                    continue
                typ = {"tsdf": "<f2", "weight": "<i2"}[key] if half else "<f4"
                self.read[key] = device_tensor(getattr(view, key), (n, 512), typ)[order]
                self.read[key] = _padded(self.read[key], self.rows)
            if half:  # unsigned 16-bit weights
                self.read["weight"] = self.read["weight"].int() & 0xFFFF
        return self.read[name]


class _Mesh(dict):
    """An extracted mesh, read when it is looked at: triangles by ascending
    vertex positions (blocks emit in no fixed order)."""

    def __init__(self, state, n):
        self.state, self.n, self.read = state, n, None
        super().__init__((k, None) for k in ["vertices", "posnor"] + ["rgb"] * (state["rgb"] is not None))

    def __getitem__(self, name):
        if self.read is None:
            torch.cuda.synchronize()
            tri = self.state["posnor"][: self.n].reshape(-1, 18)
            order = torch.arange(tri.shape[0], device=tri.device)
            for c in (14, 13, 12, 8, 7, 6, 2, 1, 0):
                order = order[torch.argsort(tri[order, c], stable=True)]
            self.read = {"vertices": self.n, "posnor": _padded(tri[order], MESH_VERTS // 3)}
            if self.state["rgb"] is not None:
                self.read["rgb"] = _padded(self.state["rgb"][: self.n].reshape(-1, 9)[order], MESH_VERTS // 3)
        return self.read[name]


# ---- the pass --------------------------------------------------------------

def _volume(case):
    vol = CudaVolume(case["voxel"], case["pool"], case["trunc"] * case["voxel"], case["cap"],
                     storage=STORAGE[case["storage"]])
    if case["pipelined"]:
        vol.set_pipelined(True)
    return vol


def _calls(case, seed):
    """The calls of one pass, each as (points or images, per-call arguments)."""
    n, per = case["frames"], case["per_call"]
    if case["source"] == "depth":
        depth, Rs, ts, K = _frames(seed, case["width"], case["height"], n)
        return [(depth[k:k + per], (K, Rs[k:k + per], ts[k:k + per])) for k in range(0, n, per)]
    clouds, cams = _clouds(seed, case["width"], case["height"], n)
    calls = []
    for k in range(0, n, per):
        part = clouds[k:k + per]
        begin = np.concatenate([[0], np.cumsum([p.shape[0] for p in part])]).astype(np.int32)
        calls.append((torch.cat(part), (begin, cams[k:k + per])))
    return calls


def _integrate(case, vol, calls):
    radius = case["radius"]
    for data, args in calls:
        if case["source"] == "depth":
            K, R, t = args
            if data.shape[0] == 1:
                vol.integrate_depth(data[0], K, R[0], t[0])
            else:
                vol.integrate_depth_frames(data, K, R, t)
        elif case["source"] == "split":
            vol.allocate_blocks(data, args[1][0], radius)
            vol.update_voxels(data, args[1][0], radius)
        elif len(args[1]) == 1:
            vol.integrate(data, args[1][0], radius)
        else:
            vol.integrate_frames(data, args[0], args[1], radius)


def prepare(case, seed):
    if case["kind"] == "batch":
        sizes = _scene_sizes(case)
        state = {"case": case, "vols": [], "frames": [], "batch": Batch(len(sizes))}
        for i, (w, h, voxel, pool) in enumerate(sizes):
            vol = CudaVolume(voxel, pool, 4.0 * voxel, case["cap"], storage=STORAGE[case["storage"]])
            clouds, cams = _clouds(seed + 101 * i, w, h, case["frames"])
            state["batch"].add(vol, w * h)
            state["vols"].append(vol)
            state["frames"].append(list(zip(clouds, cams)))
        state["batch"].set_graph(True)
        return state
    state = {"case": case, "calls": _calls(case, seed), "vol": _volume(case)}
    vol = state["vol"]
    if case["kind"] == "live":
        for _ in range(case["laps"]):
            _integrate(case, vol, state["calls"])
        vol.synchronize()
    elif case["kind"] == "extract":
        _integrate(case, vol, state["calls"])
        vol.synchronize()
        state["calls"] = None
        state["posnor"] = torch.empty((MESH_VERTS, 6), dtype=torch.float32, device="cuda")
        state["rgb"] = torch.empty((MESH_VERTS, 3), dtype=torch.uint8, device="cuda") if case["rgb"] else None
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        batch, vols = state["batch"], state["vols"]
        batch.synchronize()
        for vol in vols:
            vol.reset()
        for k in range(case["frames"]):
            for i, frames in enumerate(state["frames"]):
                batch.set_frame(i, frames[k][0], frames[k][1])
            batch.step()
        return [_Blocks(vol, state, _rows(voxel, 4.0, pool))
                for vol, (_, _, voxel, pool) in zip(vols, _scene_sizes(case))]
    vol = state["vol"]
    if case["kind"] == "extract":
        return _Mesh(state, vol.extract_mesh_device(state["posnor"], state["rgb"]))
    if case["kind"] == "session":
        vol.reset()
    _integrate(case, vol, state["calls"])
    return _Blocks(vol, state, _rows(case["voxel"], case["trunc"], case["pool"]))


# ---- what a pass computes, in plain torch ----------------------------------

def _walk(points, cam, voxel, trunc, radius):
    """The band samples of one frame in (point, step) order: the key of every
    sample's voxel (-1: none) and its normalised signed distance in 64 bits.
    Positions and voxels round as the float32 walk does; distances are double."""
    f = lambda x: torch.tensor(float(np.float32(x)), dtype=torch.float32, device=points.device)  # noqa: E731
    vs, tr = np.float32(voxel), np.float32(trunc)
    inv = np.float32(1.0) / vs
    steps = max(1, int(np.ceil(tr * inv)))
    cam32 = [f(c) for c in cam]
    d = [points[:, i] - cam32[i] for i in range(3)]
    d2 = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2]
    dist = d2.sqrt()
    live = dist > 1e-6
    if radius > 0:
        live &= d2 <= f(np.float32(radius) * np.float32(radius))
    unit = [c / dist for c in d]
    d64 = [points[:, i].double() - float(np.float32(cam[i])) for i in range(3)]
    dist64 = ((d64[0] * d64[0] + d64[1] * d64[1]) + d64[2] * d64[2]).sqrt()
    keys, vals = [], []
    for s in range(-steps, steps + 1):
        t = f(np.float32(s) * vs)
        vox = [torch.floor((points[:, i] + unit[i] * t) * f(inv)) for i in range(3)]
        e = [(vox[i] + 0.5) * f(vs) - cam32[i] for i in range(3)]
        sdf = dist - ((e[0] * e[0] + e[1] * e[1]) + e[2] * e[2]).sqrt()
        ok = live & ~(sdf < f(-tr))
        c = [vox[i].long() for i in range(3)]
        key = 0
        for x in c:
            key = (key << 18) + ((x >> 3) + (1 << 17))
        key = (key << 9) + (((c[2] & 7) << 6) + ((c[1] & 7) << 3) + (c[0] & 7))
        keys.append(torch.where(ok, key, torch.full_like(key, -1)))
        e64 = [(vox[i].double() + 0.5) * float(vs) - float(np.float32(cam[i])) for i in range(3)]
        sdf64 = dist64 - ((e64[0] * e64[0] + e64[1] * e64[1]) + e64[2] * e64[2]).sqrt()
        vals.append((sdf64 / float(tr)).clamp(-1.0, 1.0))
    return torch.stack(keys, 1).reshape(-1), torch.stack(vals, 1).reshape(-1)


def _map(frames, voxel, trunc, cap, radius, laps, half, rows):
    """The map that `laps` passes over the frames [(points, cam)] leave: per
    voxel the first cap contributions count, in (pass, frame, point, step) order."""
    parts = [_walk(p, c, voxel, trunc, radius) for p, c in frames]
    key, val = torch.cat([k for k, _ in parts]), torch.cat([v for _, v in parts])
    del parts
    key, order = torch.sort(key, stable=True)
    first = int(torch.searchsorted(key, 0))  # samples without a voxel come first
    key, val = key[first:], val[order[first:]]
    del order
    vox, count = torch.unique_consecutive(key, return_counts=True)
    which = torch.repeat_interleave(torch.arange(vox.numel(), device=key.device), count)
    start = torch.cumsum(count, 0) - count
    rank = torch.arange(key.numel(), device=key.device) - start[which]
    sums = lambda v: torch.zeros(vox.numel(), dtype=torch.float64, device=key.device).index_add_(0, which, v)  # noqa: E731
    total = count * laps
    kept = total if cap <= 0 else torch.minimum(total, torch.full_like(total, math.ceil(cap)))
    rest = kept % count
    tsdf = sums(val) * (kept // count) + sums(torch.where(rank < rest[which], val, torch.zeros_like(val)))
    blocks, row = torch.unique_consecutive(vox >> 9, return_inverse=True)
    out = {}
    for name, v in (("tsdf", tsdf / kept if half else tsdf), ("weight", kept.double())):
        out[name] = torch.zeros((blocks.numel(), 512), dtype=torch.float64, device=key.device)
        out[name][row, vox & 511] = v
        out[name] = _padded(out[name], rows)
    whole = {"blocks": None, "coords": None, "dropped": None}
    if half:
        return {**whole, "tsdf": out["tsdf"], "weight": None}
    colour = 128.0 * out["weight"]
    return {**whole, **out, "r": colour, "g": colour, "b": colour}


def _case_frames(case, seed):
    clouds, cams = _clouds(seed, case["width"], case["height"], case["frames"])
    return list(zip(clouds, cams))


def exact(case, seed):
    if case["kind"] == "extract":
        return None  # which side of the surface a corner is on depends on the map's last bit
    if case["kind"] == "batch":
        return [_map(list(zip(*_clouds(seed + 101 * i, w, h, case["frames"]))), voxel, 4.0 * voxel, case["cap"],
                     0.0, 1, case["storage"] == "fp16", _rows(voxel, 4.0, pool))
                for i, (w, h, voxel, pool) in enumerate(_scene_sizes(case))]
    return _map(_case_frames(case, seed), case["voxel"], case["trunc"] * case["voxel"], case["cap"], case["radius"],
                1 + case["laps"], case["storage"] == "fp16", _rows(case["voxel"], case["trunc"], case["pool"]))


def _count(frames, voxel, trunc, radius):
    """(points, band samples, blocks) of a list of frames."""
    points = samples = 0
    blocks = torch.empty(0, dtype=torch.int64, device=_device())
    for p, c in frames:
        key, _ = _walk(p, c, voxel, trunc, radius)
        points, samples = points + p.shape[0], samples + key.numel()
        blocks = torch.unique(torch.cat([blocks, torch.unique(key[key >= 0] >> 9)]))
    return points, samples, blocks.numel()


def work(case):
    """Points or pixels read once; the blocks of the map written once (and read,
    where the map is kept). About 34 float operations a band sample."""
    per_voxel = lambda storage: 4 if storage == "fp16" else 20  # noqa: E731
    if case["kind"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for i, (w, h, voxel, _) in enumerate(_scene_sizes(case)):
            frames = list(zip(*_clouds(101 * i, w, h, case["frames"])))
            points, samples, blocks = _count(frames, voxel, 4.0 * voxel, 0.0)
            total["bytes"] += 12.0 * points + 512.0 * per_voxel(case["storage"]) * blocks
            total["flops"] += 34.0 * samples
        return total
    if case["kind"] == "extract":
        state = prepare(case, 0)
        verts, blocks = run(state).n, state["vol"].block_count()
        read = 512.0 * (4 if case["storage"] == "fp16" else 8) * blocks
        return {"bytes": read + verts * (27.0 if case["rgb"] else 24.0), "flops": 40.0 * verts}
    points, samples, blocks = _count(_case_frames(case, 0), case["voxel"], case["trunc"] * case["voxel"],
                                     case["radius"])
    inputs = 4.0 * case["width"] * case["height"] * case["frames"] if case["source"] == "depth" else 12.0 * points
    moved = 512.0 * per_voxel(case["storage"]) * blocks
    if case["kind"] == "live":
        moved += 512.0 * (4 if case["storage"] == "fp16" else 8) * blocks
    return {"bytes": inputs + moved, "flops": 34.0 * samples}
