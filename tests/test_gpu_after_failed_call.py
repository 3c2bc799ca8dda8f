"""A call that fails with a CUDA error (here a map larger than the device) reports
it once: the next call on another map, whose launches are checked through the
runtime's last error, does what it would have done. (A reset that stopped at
that check had cleared the index and not the counters.)"""
import numpy as np
import pytest
import torch

from voxelmapping_b200 import MapBatch, VoxelMapping, synth
from voxelmapping_b200 import _lib as L
from common import block_keys, to_gpu_depth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]


def new_map(blocks):
    vm = VoxelMapping(WL.width, WL.height, WL.K, voxel_format="f32", with_color=False)
    vm.CreateMap(8, blocks, WL.voxel_size)
    return vm


def fuse(vm, i):
    d, _, pose = synth.Scene(WL).render(i)
    vm.FuseDepth(to_gpu_depth(d), pose)
    return pose


def blocks(vm):
    e = vm.export_blocks()
    i = np.argsort(block_keys(e["coords"]))
    return [e[k][i] for k in ("coords", "tsdf", "weight")]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(blocks(a), blocks(b)))


@pytest.fixture
def failed():
    def call():
        with pytest.raises(L.VmapError):
            new_map(1 << 29)  # 2.2 TB
    return call


def test_reset(failed):
    vm, want = new_map(1 << 14), new_map(1 << 14)
    fuse(vm, 0)
    failed()
    vm.reset()
    assert vm.stats()["allocated_blocks"] == 0
    fuse(vm, 40)
    fuse(want, 40)
    assert same(vm, want)


def test_snapshot_mesh_and_export(failed):
    vm = new_map(1 << 14)
    pose = fuse(vm, 0)
    failed()
    snap = vm.save_snapshot()
    other = new_map(1 << 14)
    failed()
    other.load_snapshot(snap)
    assert same(vm, other)
    failed()
    n, verts, norms = vm.Polygonize()
    assert n > 1000 and len(verts) == n
    failed()
    assert len(vm.export_blocks_static(0, 16)["coords"]) == 16
    failed()
    v = vm.RenderScene(None, pose).cpu().numpy()
    b = MapBatch([other])
    out = torch.full((WL.height, WL.width, 4), float("nan"), device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    failed()
    b.step([None], None, [pose], [out], stream=s.cuda_stream)
    s.synchronize()
    assert np.array_equal(v, out.cpu().numpy(), equal_nan=True) and np.isfinite(v).any()
    b.release()
