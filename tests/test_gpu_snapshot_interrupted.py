"""A snapshot load that stopped half-way (counters cleared, copies done or not,
index not rebuilt) leaves old voxels in the pool that no counter tells of. A
reset, or the next load, must clear them: blocks handed out afterwards start
unobserved. The state such a load leaves is written into a map that lives in
caller memory."""
import numpy as np
import pytest
import torch

from common import block_keys, to_gpu_depth
from voxelmapping_b200 import VoxelMapping, synth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]
BLOCKS, BUCKETS = 1 << 14, 1 << 14
COUNTERS, UNKNOWN = 16, 10  # words of the counter array; the one set while a load runs


def up(n):
    return -(-n // 256) * 256


def map_in_memory():
    vm = VoxelMapping(WL.width, WL.height, WL.K, voxel_format="f32", with_color=False, num_buckets=BUCKETS)
    mem = torch.zeros(vm.required_bytes(8, BLOCKS, WL.voxel_size), dtype=torch.uint8, device="cuda")
    vm.CreateMapIn(8, BLOCKS, WL.voxel_size, mem)
    return vm, mem


def fuse(vm, scene, idx):
    for i in idx:
        d, _, pose = scene.render(i)
        vm.FuseDepth(to_gpu_depth(d), pose)


def interrupt(mem):
    """The counters as a load leaves them that fails before it rebuilds the index."""
    at = up(BUCKETS * 4 * 16) + up(BLOCKS * 28) + up(BLOCKS * 8) + up(BLOCKS * 512 * 8)
    ctr = mem[at:at + 4 * COUNTERS].view(torch.int32)
    assert int(ctr[0]) > 1000  # the blocks allocated
    ctr[:UNKNOWN] = 0
    ctr[UNKNOWN] = 0x01010101


def same(a, b):
    ea, eb = a.export_blocks(), b.export_blocks()
    ia, ib = np.argsort(block_keys(ea["coords"])), np.argsort(block_keys(eb["coords"]))
    for k in ("coords", "tsdf", "weight"):
        assert np.array_equal(ea[k][ia], eb[k][ib]), k


@pytest.mark.parametrize("then", ["reset", "load", "load and reset", "load of nothing"])
def test_blocks_start_unobserved_after_an_interrupted_load(then):
    scene = synth.Scene(WL)
    vm, mem = map_in_memory()
    fresh, _ = map_in_memory()
    small, _ = map_in_memory()
    if then != "load of nothing":
        d, _, pose = scene.render(40)
        d[:, WL.width // 4:] = 0
        small.FuseDepth(to_gpu_depth(d), pose)
    snap = small.save_snapshot()
    fuse(vm, scene, (0, 10, 20))
    assert vm.stats()["allocated_blocks"] > small.stats()["allocated_blocks"] + 1000
    interrupt(mem)
    if then.startswith("load"):
        vm.load_snapshot(snap)
        fresh.load_snapshot(snap)
    if then.endswith("reset"):
        if then == "load and reset":
            fuse(vm, scene, (40,))
        vm.reset()
        fresh.reset()
    for m in (vm, fresh):
        fuse(m, scene, (30, 60))
    assert vm.stats()["error_flags"] == 0
    same(vm, fresh)
