"""The block grid behind the ray marcher's lookups changes no result: maps of
different capacity (grids of 16 to 128 cells per axis, with and without two blocks in
one cell, and no grid) and maps far from the origin (the ray marcher's wide
form) render, bit for bit, what a large map does; and a reset or a loaded
snapshot leaves no stale entry."""
import numpy as np
import pytest

from voxelmapping_b200 import MapBatch, VoxelMapping, synth
from common import to_gpu_depth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]
W, H = 161, 119
K = np.array([[132.0, 0, 80.0], [0, 132.0, 59.0], [0, 0, 1]])


def new_map(blocks, fmt="f32", mode=0, vs=0.016):
    vm = VoxelMapping(W, H, K, voxel_format=fmt, with_color=False, raycast_mode=mode)
    vm.CreateMap(4 * blocks, blocks, vs)
    return vm


def frames(n, shift):
    """Depth crops and poses of the room, moved by `shift` metres."""
    sc = synth.Scene(WL)
    out = []
    for i in range(n):
        d, _, pose = sc.render(3 * i)
        p = pose.copy()
        p[:3, 3] += shift
        out.append((to_gpu_depth(np.pad(d[::2, ::2], ((0, 0), (0, 1)))[:H, :W]), p))
    return out


def drive(vm, fs, poses):
    import torch
    for d, p in fs:
        vm.FuseDepth(d, p)
    out = []
    for p in poses:
        n = torch.empty((H, W, 4), device="cuda")
        v = vm.RenderScene(None, p, n)
        out += [v.cpu().numpy(), n.cpu().numpy()]
    assert vm.stats()["error_flags"] == 0
    return out


def same(a, b):
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))
    assert sum(int(np.isfinite(x).sum()) for x in a) > 1000


# shift in metres: at 16 mm the narrow range ends at 1,032 m (2^12 blocks, 16 cells on the shortest axis), 2,080 m
# (2^15, 32) and 4,178 m (2^18, 64)
@pytest.mark.parametrize("shift", [0.0, -900.0, 1500.0, 3000.0, -5000.0])
@pytest.mark.parametrize("mode", [0, 1])
def test_capacities_agree(shift, mode):
    fs = frames(2, np.array([shift, -0.5 * shift, 0.25 * shift]))
    poses = [fs[1][1], fs[0][1]]
    want = drive(new_map(1 << 18, mode=mode), fs, poses)
    for blocks in (1 << 12, 1 << 15):
        same(drive(new_map(blocks, mode=mode), fs, poses), want)


@pytest.mark.parametrize("fmt", ["ref", "f16", "i16"])
def test_formats_and_shared_cells(fmt):
    """4 mm voxels: the room spans 125 blocks, more than the smaller grid's 64 x 32 x 32 cells."""
    fs = [(d, p) for d, p in frames(1, np.zeros(3))]
    poses = [fs[0][1]]
    want = drive(new_map(1 << 18, fmt, vs=0.004), fs, poses)
    same(drive(new_map(1 << 15, fmt, vs=0.004), fs, poses), want)


def test_reset_and_snapshot_leave_no_stale_entry():
    fs, gs = frames(1, np.zeros(3)), frames(1, np.array([0.7, 0.3, 0.0]))
    want = drive(new_map(1 << 13), gs, [gs[0][1], fs[0][1]])
    vm = new_map(1 << 13)
    drive(vm, fs, [fs[0][1]])
    snap = vm.save_snapshot()
    vm.reset()
    same(drive(vm, gs, [gs[0][1], fs[0][1]]), want)
    vm.load_snapshot(snap)
    same(drive(vm, [], [fs[0][1]]), drive(new_map(1 << 12), fs, [fs[0][1]]))


def test_batch_with_a_far_map_takes_the_wide_form():
    import torch
    near, far = frames(2, np.zeros(3)), frames(2, np.full(3, 4900.0))
    maps = [new_map(1 << 13), new_map(1 << 13)]
    solo = [drive(new_map(1 << 13), [f[0]], [f[0][1]]) for f in (near, far)]
    b = MapBatch(maps)
    v, n = ([torch.empty((H, W, 4), device="cuda") for _ in maps] for _ in range(2))
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    b.step([f[0][0] for f in (near, far)], None, [f[0][1] for f in (near, far)], v, n, stream=s.cuda_stream)
    s.synchronize()
    for i in range(2):
        same([v[i].cpu().numpy(), n[i].cpu().numpy()], solo[i])
    # the same batch without the far map's render: the narrow form, another graph
    for _ in range(3):
        b.step([near[1][0], None], None, [near[1][1], far[0][1]], [v[0], None], [n[0], None], stream=s.cuda_stream)
    s.synchronize()
    m = new_map(1 << 13)
    drive(m, [near[0]] + [near[1]] * 3, [])
    w = torch.empty((H, W, 4), device="cuda")
    same([v[0].cpu().numpy(), n[0].cpu().numpy()], [m.RenderScene(None, near[1][1], w).cpu().numpy(), w.cpu().numpy()])


def test_tiny_map_without_a_grid():
    import torch
    d = torch.zeros((H, W), dtype=torch.int16, device="cuda")
    d[60:66, 80:86] = 1000
    out = []
    for blocks in (8, 1 << 12):
        vm = VoxelMapping(W, H, K, voxel_format="f32", with_color=False)
        vm.CreateMap(0, blocks, 0.016)
        for _ in range(3):
            vm.FuseDepth(d, np.eye(4))
        p = np.eye(4)
        p[0, 3] = 0.01
        out.append([vm.RenderScene(None, x).cpu().numpy() for x in (np.eye(4), p)])
        st = vm.stats()
        assert st["error_flags"] == 0 and 0 < st["allocated_blocks"] <= 8
    assert np.isfinite(out[0][0]).any()
    assert all(np.array_equal(a, b, equal_nan=True) for a, b in zip(*out))
