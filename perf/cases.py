"""Timed cases: what a user of this library has it do, through its public
entry points, over the sizes, storage formats and options it is used with.

Every case works in a box room with spheres seen from inside, the scene of the
library's own workloads (room_small: 320x240, 8 mm voxels, int16 storage;
room_full: 640x480, 5 mm, FP32 + colour): uint16 millimetre depth with axial
noise and 2 % dropouts, a camera on a figure-8. Frames are made on the GPU from
the seed alone. A map that a program already holds has fused every fifth frame
of the lap so far.

  track   one frame of a tracking loop: fuse depth (+ colour), then render the
          vertex and normal maps the next frame is registered against
  views   candidate poses rendered without normals, as for relocalisation
  viewer  a free view with normals and its Phong picture, beside the normals
          and picture of the live frame
  start   a session begins: the map is emptied, the first frame fused, rendered
  batch   one step of many maps, every one with its own frame
  mesh    all triangles and normals of a map, and their centroids
  swap    a session comes back from host memory, takes a frame, is evicted
  host    frames from host memory through the pipelined host path

`exact` gives the live normals of `viewer` in 64 bits. The other floating
outputs have no such value: a ray's samples, its hit or miss and a voxel's
pixel are decided by single-precision comparisons (floor, sign, step counts),
so a 64-bit run decides some of them otherwise and has misses elsewhere.
"""
import ctypes
import math
import random

import numpy as np
import torch

from voxelmapping_b200 import _lib
from voxelmapping_b200.vmapping import HostPipeline, MapBatch, VoxelMapping

DEPTH_SCALE = 0.001
LAP = 500  # poses of one lap


def listed():
    c = []
    # the smallest call: a robot's low-resolution depth camera on coarse voxels
    c.append(dict(name="track_160x120", op="track", w=160, h=120, voxel=0.016, fmt="ref", color=False, depth="f32",
                  room=4.0, blocks=1 << 14, prefix=20))
    # room_small: the reference's own storage and its float depth input
    c.append(dict(name="track_320x240", op="track", w=320, h=240, voxel=0.008, fmt="ref", color=False, depth="f32",
                  room=4.0, blocks=1 << 18, prefix=20))
    # room_full: the ordinary RGB-D frame, FP32 + colour
    c.append(dict(name="track_640x480", op="track", w=640, h=480, voxel=0.005, fmt="f32", color=True, depth="u16",
                  room=4.0, blocks=1 << 20, prefix=20))
    # the largest camera of the uneven mix at its finest voxels, half storage
    c.append(dict(name="track_1280x720", op="track", w=1280, h=720, voxel=0.004, fmt="f16", color=True, depth="u16",
                  room=6.0, blocks=1 << 19, prefix=20))
    # relocalisation on a cropped image: eight candidate poses, no normals
    c.append(dict(name="views_517x389", op="views", w=517, h=389, voxel=0.006, fmt="i16", color=False, depth="u16",
                  room=4.0, blocks=1 << 17, prefix=20, views=8, mode=0))
    # a viewer with the reference's full march from 0.1 m
    c.append(dict(name="viewer_800x600", op="viewer", w=800, h=600, voxel=0.008, fmt="f32", color=True, depth="u16",
                  room=4.0, blocks=1 << 18, prefix=20, mode=1))
    # a session's first frame on a map that was in use
    c.append(dict(name="start_640x480", op="start", w=640, h=480, voxel=0.005, fmt="f32", color=True, depth="u16",
                  room=4.0, blocks=1 << 20, prefix=0))
    # a server's tick: equal sessions, then a mix of cameras and voxel sizes
    c.append(dict(name="batch_32x640x480", op="batch", maps=32, mixed=False, w=640, h=480, voxel=0.005, fmt="f16",
                  color=True, depth="u16", room=4.0, blocks=1 << 16, prefix=8))
    c.append(dict(name="batch_48_mixed", op="batch", maps=48, mixed=True, w=320, h=240, voxel=0.008, fmt="i16",
                  color=True, depth="u16", room=4.0, blocks=1 << 16, prefix=8))
    # the mesh of a room after a lap
    c.append(dict(name="mesh_room", op="mesh", w=640, h=480, voxel=0.008, fmt="f32", color=True, depth="u16",
                  room=4.0, blocks=1 << 18, prefix=60))
    # a served session under memory pressure
    c.append(dict(name="swap_320x240", op="swap", w=320, h=240, voxel=0.008, fmt="f16", color=True, depth="u16",
                  room=4.0, blocks=1 << 14, prefix=12))
    # a camera's frames from host memory, results back to the host
    c.append(dict(name="host_640x480", op="host", w=640, h=480, voxel=0.005, fmt="f32", color=True, depth="u16",
                  room=4.0, blocks=1 << 18, prefix=12, frames=4))
    return c


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    op = rng.choice(["track"] * 5 + ["views", "viewer", "start", "batch", "mesh", "swap", "host"])
    c = dict(op=op, fmt=rng.choice(["ref", "f32", "f16", "i16"]), color=rng.random() < 0.5,
             depth=rng.choice(["f32", "u16"]), room=round(_log(rng, 2.0, 6.0), 2), voxel=round(_log(rng, 0.004, 0.016), 4))
    c["w"] = int(round(_log(rng, 96, 1280 if op == "track" else 800)))
    c["h"] = int(round(c["w"] * rng.uniform(0.55, 0.8)))
    c["prefix"] = {"start": 0, "batch": 8, "mesh": 40}.get(op, rng.randint(8, 20))
    if op == "views":
        c["views"] = rng.randint(1, 8)
    if op in ("views", "viewer"):
        c["mode"] = rng.randint(0, 1)
    if op == "host":
        c["frames"] = rng.randint(1, 4)
    if op == "mesh":
        c["voxel"] = max(c["voxel"], 0.007)
    if op == "swap":
        c["voxel"] = max(c["voxel"], 0.01)
    if op == "batch":
        c["maps"] = int(round(_log(rng, 2, 48)))
        c["mixed"] = rng.random() < 0.5
        c["w"] = int(round(_log(rng, 80, 320)))
        c["h"] = int(round(c["w"] * 0.75))
        c["voxel"] = max(c["voxel"], 0.006)
    # twice the blocks of the room's surface, as the uneven workloads size their pools
    c["blocks"] = 1 << int(min(15 if op == "swap" else 19, max(13, math.ceil(math.log2(3.0 * _area(c) / (8 * c["voxel"]) ** 2)))))
    return c


# ------------------------------------------------------------------ the scene
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _height(room):
    return min(3.0, 0.75 * room)


def _area(c):
    """The room's surface in square metres."""
    return 2.0 * (c["room"] ** 2 + 2 * c["room"] * _height(c["room"]))


class _Scene:
    """A room of `room` x `room` metres with 8 spheres clear of the camera's path."""

    def __init__(self, room, seed):
        rng = random.Random(seed)
        self.hx, self.hz = room / 2, _height(room)
        self.r, self.z = room / 4, self.hz / 2
        self.spheres = []
        while len(self.spheres) < 8:
            rad = rng.uniform(0.1, 0.5) * min(1.0, room / 4)
            x, y = (rng.uniform(rad - self.hx, self.hx - rad) for _ in range(2))
            z = rng.uniform(rad, self.hz - rad)
            if abs(z - self.z) > rad + 0.25 or math.hypot(x, y) > self.r + rad + 0.25 or rng.random() < 0.02:
                self.spheres.append((x, y, z, rad))
        self.colours = [[rng.randrange(40, 240) for _ in range(3)] for _ in range(14)]
        self.phase = rng.uniform(0.0, 2 * math.pi)

    def pose(self, k, turn=0.0):
        """Camera-to-world pose k of the lap (OpenCV axes), `turn` further along the target's circle."""
        t = self.phase + 2 * math.pi * k / LAP
        pos = np.array([self.r * math.sin(t), self.r * math.sin(t) * math.cos(t), self.z + 0.1 * self.r * math.sin(3 * t)])
        tgt = np.array([1.5 * self.r * math.cos(t + turn), 1.5 * self.r * math.sin(t + turn), self.z - 0.2 * self.r])
        f = (tgt - pos) / np.linalg.norm(tgt - pos)
        right = np.cross(f, [0.0, 0.0, 1.0])
        right /= np.linalg.norm(right)
        T = np.eye(4)
        T[:3, 0], T[:3, 1], T[:3, 2], T[:3, 3] = right, np.cross(f, right), f, pos
        return T

    def frames(self, poses, c, gen):
        """Depth (n, h, w) in millimetres (int16 holding uint16) and colour (n, h, w, 3) of the poses."""
        dev, w, h, f = _device(), c["w"], c["h"], 0.8203125 * c["w"]
        T = torch.tensor(np.stack(poses), dtype=torch.float64, device=dev)
        u = (torch.arange(w, dtype=torch.float64, device=dev) - (w - 1) / 2) / f
        v = (torch.arange(h, dtype=torch.float64, device=dev) - (h - 1) / 2) / f
        rays = [T[:, i, 0, None, None] * u[None, None, :] + T[:, i, 1, None, None] * v[None, :, None] + T[:, i, 2, None, None]
                for i in range(3)]
        o = [T[:, i, 3, None, None] for i in range(3)]
        depth, what = torch.full_like(rays[0], 1e30), torch.zeros(rays[0].shape, dtype=torch.int64, device=dev)
        for i, (lo, hi) in enumerate(((-self.hx, self.hx), (-self.hx, self.hx), (0.0, self.hz))):
            up = rays[i] > 0
            t = torch.where(up, hi - o[i], lo - o[i]) / rays[i]
            near = (rays[i].abs() > 1e-12) & (t < depth)
            depth, what = torch.where(near, t, depth), torch.where(near, 2 * i + up.long(), what)
        a = rays[0] ** 2 + rays[1] ** 2 + rays[2] ** 2
        for k, (x, y, z, rad) in enumerate(self.spheres):
            oc = (o[0] - x, o[1] - y, o[2] - z)
            b = oc[0] * rays[0] + oc[1] * rays[1] + oc[2] * rays[2]
            disc = b * b - a * (oc[0] ** 2 + oc[1] ** 2 + oc[2] ** 2 - rad * rad)
            t = (-b - disc.clamp(min=0).sqrt()) / a
            near = (disc > 0) & (t > 1e-9) & (t < depth)
            depth, what = torch.where(near, t, depth), torch.where(near, 6 + k, what)
        noise = torch.randn(depth.shape, dtype=torch.float64, device=dev, generator=gen)
        depth = depth + noise * (0.0012 + 0.0019 * (depth - 0.4) ** 2)
        depth = torch.where(torch.rand(depth.shape, device=dev, generator=gen) < 0.02, torch.zeros_like(depth), depth)
        mm = (depth * 1000.0).round().clamp(0, 32767).to(torch.int16)
        rgb = torch.tensor(self.colours, dtype=torch.uint8, device=dev)[what] if c["color"] else None
        return mm, rgb


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _sensor(c, mm):
    """The depth image as the camera's driver hands it over: uint16 millimetres or float metres."""
    return mm if c["depth"] == "u16" else mm.to(torch.float32) * DEPTH_SCALE


# -------------------------------------------------------------------- the map
def _new_map(c):
    f = 0.8203125 * c["w"]
    K = [[f, 0, (c["w"] - 1) / 2], [0, f, (c["h"] - 1) / 2], [0, 0, 1]]
    vm = VoxelMapping(c["w"], c["h"], K, voxel_format=c["fmt"], with_color=c["color"], raycast_mode=c.get("mode", 0))
    vm.CreateMap(2 * c["blocks"], c["blocks"], c["voxel"])
    return vm


def _fuse(vm, frame):
    depth, rgb, pose = frame
    if rgb is None:
        vm.FuseDepth(depth, pose, DEPTH_SCALE)
    else:
        vm.FuseDepthAndImage(rgb, depth, pose, DEPTH_SCALE)


def _frames(c, scene, gen, ks):
    """[(depth, rgb or None, pose)] of the lap's poses ks."""
    poses = [scene.pose(k) for k in ks]
    mm, rgb = scene.frames(poses, c, gen)
    d = _sensor(c, mm)
    return [(d[i], rgb[i] if rgb is not None else None, poses[i]) for i in range(len(poses))]


def _image(c):
    return torch.full((c["h"], c["w"], 4), float("nan"), dtype=torch.float32, device="cuda")


def _of_map(c, i):
    """Map i of a batch: in a mixed one the cameras are half, one and twice the size, the voxels 1 to 2 times as large."""
    if not c["mixed"]:
        return dict(c)
    s = (0.5, 1.0, 2.0)[i % 3]
    return dict(c, w=max(48, int(c["w"] * s)), h=max(36, int(c["h"] * s)), voxel=c["voxel"] * (1.0, 1.25, 1.5, 2.0)[i % 4])


def _sorted_snapshot(vm):
    """The map's snapshot with its blocks in the order of their keys: blocks are
    handed out in whatever order threads reach them, and a snapshot keeps it."""
    raw = vm.save_snapshot(torch.empty(vm.snapshot_bytes(), dtype=torch.uint8, device="cuda"))
    h = _lib.SnapshotHeader.from_buffer_copy(bytes(raw[:ctypes.sizeof(_lib.SnapshotHeader)].cpu().numpy()))
    keys = raw[h.keys_offset:h.keys_offset + 8 * h.n_blocks]
    pool = raw[h.pool_offset:].view(h.n_blocks, h.block_bytes)
    order = torch.argsort(keys.clone().view(torch.int64))
    out = raw.clone()
    out[h.keys_offset:h.keys_offset + 8 * h.n_blocks] = keys.view(h.n_blocks, 8)[order].reshape(-1)
    out[h.pool_offset:] = pool[order].reshape(-1)
    return out


def prepare(case, seed):
    c, gen = dict(case), _gen(seed)
    op, n = c["op"], c["prefix"]
    if op == "batch":
        s = dict(case=c, maps=[], frames=[], at=0)
        every = [_of_map(c, i) for i in range(c["maps"])]
        sizes = sorted({(ci["h"], ci["w"]) for ci in every})
        # the maps of one camera size render into one array
        same = {z: [i for i, ci in enumerate(every) if (ci["h"], ci["w"]) == z] for z in sizes}
        for what in ("vmap", "nmap"):
            s[what] = [torch.full((len(same[z]), *z, 4), float("nan"), dtype=torch.float32, device="cuda") for z in sizes]
            at = {i: s[what][k][j] for k, z in enumerate(sizes) for j, i in enumerate(same[z])}
            s[what + "s"] = [at[i] for i in range(c["maps"])]
        for i, ci in enumerate(every):
            scene = _Scene(c["room"], seed * 1009 + i)
            got = _frames(ci, scene, gen, [5 * k for k in range(n)] + [5 * n, 5 * n + 1])
            vm = _new_map(ci)
            for f in got[:n]:
                _fuse(vm, f)
            s["maps"].append(vm)
            s["frames"].append([(d.clone(), r.clone() if r is not None else None, p) for d, r, p in got[n:]])
        s["batch"] = MapBatch(s["maps"])
        s["stream"] = torch.cuda.Stream()
        torch.cuda.synchronize()  # the step runs on a stream of its own
        return s
    scene = _Scene(c["room"], seed)
    stride = 12 if op == "mesh" else 5
    # a session's frame on eviction is one it has seen the like of: the map does not grow
    last = [n * 5 - 5] if op == "swap" else [n * stride + k for k in range(4)]
    ks = [stride * k for k in range(n)]
    got = _frames(c, scene, gen, ks + ([] if op == "swap" else last))
    vm = _new_map(c)
    for f in got[:n]:
        _fuse(vm, f)
    s = dict(case=c, vm=vm, at=0, frames=[(d.clone(), r.clone() if r is not None else None, p) for d, r, p in got[-4:]],
             vmap=_image(c), nmap=_image(c))
    if op == "swap":
        snap = _sorted_snapshot(vm)
        s["snap"] = torch.empty(snap.numel(), dtype=torch.uint8).pin_memory()
        s["snap"].copy_(snap)
        # room for the snapshot of a full pool
        most = 256 + 8 * c["blocks"] + 256 + c["blocks"] * int(vm._lib.vmap_block_bytes(vm.voxel_format, int(c["color"])))
        s["out"] = torch.zeros(most, dtype=torch.uint8).pin_memory()
    elif op == "views":
        s["poses"] = [scene.pose(5 * n - 3 * k, 0.05 * (k % 3)) for k in range(c["views"])]
        s["vmaps"] = [_image(c) for _ in range(c["views"])]
    elif op == "viewer":
        s["pose"] = scene.pose(4 * n, 0.1)
        s["image"], s["live_image"] = (torch.zeros((c["h"], c["w"], 4), dtype=torch.uint8, device="cuda") for _ in range(2))
        s["live"], s["live_nmap"] = _live(c, s["frames"][0][0]), _image(c)
    elif op == "mesh":
        # room for twice the triangles of the room's bare surface at this voxel size
        s["most"] = int(4 * _area(c) / c["voxel"] ** 2)
        s["count"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        for what, lanes in (("verts", 9), ("norms", 9), ("points", 3)):
            s[what], s[what + "_ordered"] = (torch.zeros((s["most"], lanes), device="cuda") for _ in range(2))
        s["mix"] = torch.tensor([random.Random(k).getrandbits(62) * 2 + 1 for k in range(9)], device="cuda")
    elif op == "host":
        s["pipe"] = HostPipeline(vm, DEPTH_SCALE)
        s["host"] = [(d.cpu().numpy().view(np.uint16) if c["depth"] == "u16" else d.cpu().numpy(),
                      r.cpu().numpy() if r is not None else None, p) for d, r, p in s["frames"]]
    torch.cuda.synchronize()
    return s


def _live(c, depth):
    """The live frame's vertex map, NaN where there is no depth."""
    w, h, f = c["w"], c["h"], 0.8203125 * c["w"]
    z = depth.to(torch.float32) * DEPTH_SCALE if c["depth"] == "u16" else depth
    z = torch.where(z > 0, z, torch.full_like(z, float("nan")))
    u = (torch.arange(w, device=z.device) - (w - 1) / 2) / f
    v = (torch.arange(h, device=z.device) - (h - 1) / 2) / f
    return torch.stack([u[None, :] * z, v[:, None] * z, z, torch.ones_like(z)], -1).contiguous()


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


# ------------------------------------------------------------------- one pass
def run(s):
    c, op = s["case"], s["case"]["op"]
    if op == "batch":
        now = [f[s["at"]] for f in s["frames"]]
        s["at"] ^= 1
        s["batch"].step([f[0] for f in now], [f[1] for f in now] if c["color"] else None, [f[2] for f in now], s["vmaps"],
                        s["nmaps"], DEPTH_SCALE, s["stream"].cuda_stream)
        return {"vmaps": s["vmap"], "nmaps": s["nmap"]}
    vm = s["vm"]
    if op in ("track", "start"):
        frame = s["frames"][s["at"]]
        s["at"] = (s["at"] + 1) % len(s["frames"])
        if op == "start":
            vm.reset()
        _fuse(vm, frame)
        vm.RenderScene(s["vmap"], frame[2], s["nmap"])
        return {"vmap": s["vmap"], "nmap": s["nmap"]}
    if op == "views":
        for pose, v in zip(s["poses"], s["vmaps"]):
            vm.RenderScene(v, pose)
        return {"vmaps": s["vmaps"]}
    if op == "viewer":
        w, h, lib = c["w"], c["h"], vm._lib
        vm.RenderScene(s["vmap"], s["pose"], s["nmap"])
        _lib.check(lib.vmap_render_phong(_ptr(s["vmap"]), 0, _ptr(s["nmap"]), 0, _ptr(s["image"]), 0, w, h, _stream()))
        _lib.check(lib.vmap_compute_normal(_ptr(s["live"]), 0, _ptr(s["live_nmap"]), 0, w, h, _stream()))
        _lib.check(lib.vmap_render_phong(_ptr(s["live"]), 0, _ptr(s["live_nmap"]), 0, _ptr(s["live_image"]), 0, w, h, _stream()))
        return {k: s[k] for k in ("vmap", "nmap", "image", "live_nmap", "live_image")}
    if op == "mesh":
        verts, norms, points, lib = s["verts"], s["norms"], s["points"], vm._lib
        _lib.check(lib.vmap_polygonize(vm._need(), None, None, 0, _ptr(s["count"]), _stream()))
        n = int(s["count"].item())
        if n > s["most"]:
            raise ValueError("%d triangles, room for %d" % (n, s["most"]))
        _lib.check(lib.vmap_polygonize(vm._need(), _ptr(verts), _ptr(norms), s["most"], _ptr(s["count"]), _stream()))
        _lib.check(lib.vmap_surface_points(_ptr(verts), n, _ptr(points), _stream()))
        # triangles come in no fixed order: a program that stores or compares meshes orders them by their contents
        order = torch.argsort((verts[:n].view(torch.int32) * s["mix"]).sum(1))
        for what in ("verts", "norms", "points"):
            torch.index_select(s[what], 0, order, out=s[what + "_ordered"][:n])
        return {what: s[what + "_ordered"] for what in ("verts", "norms", "points")}
    if op == "swap":
        vm.load_snapshot(s["snap"])
        frame = s["frames"][-1]
        _fuse(vm, frame)
        vm.RenderScene(s["vmap"], frame[2], s["nmap"])
        vm.save_snapshot(s["out"])
        return {"vmap": s["vmap"], "nmap": s["nmap"], "snapshot": s["out"]}
    out = [s["pipe"].submit(d, r, p) for d, r, p in s["host"][:c["frames"]]]
    s["pipe"].wait()
    return {"vmaps": [v for v, _ in out], "nmaps": [n for _, n in out]}


# -------------------------------------------------------------------- 64 bits
def exact(case, seed):
    if case["op"] != "viewer":
        return None
    c, n = dict(case), case["prefix"]
    got = _frames(c, _Scene(c["room"], seed), _gen(seed), [5 * k for k in range(n)] + [5 * n + k for k in range(4)])
    v = _live(c, got[-4][0])[..., :3].double()
    left, up = torch.cat([v[:, :1], v[:, :-1]], 1), torch.cat([v[:1], v[:-1]], 0)
    a = torch.cat([v[:, 1:], torch.full_like(v[:, :1], float("nan"))], 1) - left
    b = torch.cat([v[1:], torch.full_like(v[:1], float("nan"))], 0) - up
    n = torch.linalg.cross(a, b)
    size = n.norm(dim=-1, keepdim=True)
    n = torch.where(size > 0, n / size, n)
    n = torch.cat([n, torch.where(n[..., :1].isnan(), n[..., :1], torch.ones_like(n[..., :1]))], -1)
    return {"vmap": None, "nmap": None, "image": None, "live_nmap": n, "live_image": None}


# ------------------------------------------------------------------- the work
_VOXEL = {"ref": 4, "f32": 8, "f16": 4, "i16": 4}


def _blocks(c, ks):
    """Blocks that hold the surface seen from the lap's poses ks: nothing less can be read or written."""
    scene = _Scene(c["room"], 1)
    mm, _ = scene.frames([scene.pose(k) for k in ks], dict(c, color=False), _gen(1))
    f, seen = 0.8203125 * c["w"], []
    for k, d in zip(ks, mm):
        z = d.double() * DEPTH_SCALE
        u = (torch.arange(c["w"], device=z.device) - (c["w"] - 1) / 2) / f
        v = (torch.arange(c["h"], device=z.device) - (c["h"] - 1) / 2) / f
        T = torch.tensor(scene.pose(k), device=z.device)
        p = torch.stack([u[None, :] * z, v[:, None] * z, z], -1)[(z > 0.1) & (z < 5.0)] @ T[:3, :3].T + T[:3, 3]
        b = torch.floor(p / (8 * c["voxel"])).long() + (1 << 20)
        seen.append(torch.unique((b[:, 0] << 42) | (b[:, 1] << 21) | b[:, 2]))
    return int(torch.unique(torch.cat(seen)).numel())


def work(case):
    """Bytes of one pass: frames in, seen blocks once each way (once where they are only read), results out."""
    c, op = dict(case), case["op"]
    if op == "batch":
        one = [work(dict(_of_map(c, i), op="track", prefix=4)) for i in range(12 if c["mixed"] else 1)]
        return {"bytes": sum(x["bytes"] for x in one) * c["maps"] / len(one), "flops": 0.0}
    px = c["w"] * c["h"]
    voxels = 512.0 * _VOXEL[c["fmt"]]
    block = voxels + (1536.0 if c["color"] else 0.0)
    frame = px * ((2 if c["depth"] == "u16" else 4) + (3 if c["color"] else 0))
    n = c["prefix"]
    if op in ("track", "start", "swap"):
        b = frame + 2 * _blocks(c, [5 * n]) * block + 32.0 * px
        if op == "swap":
            b += 4 * _blocks(c, [5 * k for k in range(n)]) * block  # snapshot and map, in and out
    elif op == "views":
        b = c["views"] * (_blocks(c, [5 * n]) * voxels + 16.0 * px)
    elif op == "viewer":
        b = _blocks(c, [4 * n]) * voxels + px * (32.0 + 4.0 + 16.0 + 16.0 + 4.0)
    elif op == "mesh":
        got = _blocks(c, [12 * k for k in range(n)])
        b = got * voxels + got * 150.0 * (72.0 + 36.0 + 12.0)  # about 150 triangles a block with this noise
    else:
        b = c["frames"] * (frame + 2 * _blocks(c, [5 * n]) * block + 32.0 * px)
    return {"bytes": float(b), "flops": 0.0}
