"""vmap_reset clears the blocks that were handed out: a map that was used, then
reset, behaves as a new one (every format; a pool that ran full; a map that
held a snapshot of more blocks than it had itself)."""
import numpy as np
import pytest

from voxelmapping_b200 import VoxelMapping, synth
from common import block_keys, to_gpu_depth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]


def new_map(fmt="f32", color=True, blocks=1 << 14):
    vm = VoxelMapping(WL.width, WL.height, WL.K, voxel_format=fmt, with_color=color)
    vm.CreateMap(4 * blocks, blocks, WL.voxel_size)
    return vm


def fuse(vm, scene, i):
    import torch
    d, c, pose = scene.render(i)
    if vm.with_color:
        vm.FuseDepthAndImage(torch.from_numpy(c).cuda(), to_gpu_depth(d), pose)
    else:
        vm.FuseDepth(to_gpu_depth(d), pose)
    return pose


def assert_as_new(vm, scene, fmt, color, blocks):
    fresh = new_map(fmt, color, blocks)
    for m in (vm, fresh):
        pose = fuse(m, scene, 40)
    got, want = vm.export_blocks(), fresh.export_blocks()
    gi, wi = np.argsort(block_keys(got["coords"])), np.argsort(block_keys(want["coords"]))
    for k in ("coords", "tsdf", "weight") + (("rgb",) if color else ()):
        assert np.array_equal(got[k][gi], want[k][wi]), k
    v, n = vm.RenderScene(None, pose).cpu().numpy(), fresh.RenderScene(None, pose).cpu().numpy()
    assert np.array_equal(v, n, equal_nan=True)


@pytest.mark.parametrize("fmt,color", [("ref", False), ("f32", True), ("f16", True), ("i16", False)])
def test_used_map_is_as_new_after_reset(fmt, color):
    scene = synth.Scene(WL)
    vm = new_map(fmt, color)
    for i in (0, 10, 20):
        fuse(vm, scene, i)
    vm.RenderScene(None, scene.poses[20])
    vm.reset()
    assert vm.stats()["allocated_blocks"] == 0
    assert_as_new(vm, scene, fmt, color, 1 << 14)


def test_full_pool_is_cleared():
    scene = synth.Scene(WL)
    vm = new_map(blocks=300)
    fuse(vm, scene, 0)
    assert vm.stats()["failed_allocs"] > 0
    vm.reset()
    st = vm.stats()
    assert st["allocated_blocks"] == 0 and st["failed_allocs"] == 0 and st["error_flags"] == 0
    # frame 0 again hands out the whole pool: every block must start unobserved, so weights are 1
    fuse(vm, scene, 0)
    assert vm.stats()["allocated_blocks"] == 300 and vm.export_blocks()["weight"].max() == 1.0


def test_map_that_held_a_larger_snapshot():
    scene = synth.Scene(WL)
    big = new_map()
    for i in (0, 30, 60, 90):
        fuse(big, scene, i)
    vm = new_map()
    fuse(vm, scene, 0)
    vm.load_snapshot(big.save_snapshot())
    vm.reset()
    assert_as_new(vm, scene, "f32", True, 1 << 14)
