"""Both forms of the allocation against the oracle's block sets: near views (32-bit
keys, no conversions) and views that are not (voxels so small that a band is
more than 510 blocks away, cameras beyond 2^20 voxels), negative coordinates,
image sizes with remainders in both tile directions, depths at the ends of the
range, invalid depths, and a batch that mixes the two."""
import numpy as np
import pytest

from common import block_keys, to_gpu_depth
from oracle import oracle as O
from voxelmapping_b200 import MapBatch, VoxelMapping, synth

pytestmark = pytest.mark.gpu


def depth_and_pose(w, h, shift, seed):
    rng = np.random.default_rng(seed)
    d = rng.integers(60, 5200, (h, w)).astype(np.uint16)
    d[rng.random((h, w)) < 0.05] = 0
    d[0, 0] = 100  # the ends of the depth range
    d[-1, -1] = 5000
    a, b = 0.3 + seed, 0.2
    ca, sa, cb, sb = np.cos(a), np.sin(a), np.cos(b), np.sin(b)
    p = np.eye(4)
    p[:3, :3] = np.array([[ca, -sa, 0], [sa, ca, 0], [0, 0, 1]]) @ np.array([[1, 0, 0], [0, cb, -sb], [0, sb, cb]])
    p[:3, 3] = np.array([0.1, -0.2, 0.05]) + np.asarray(shift)
    return d, p


def K_of(w, h):
    return np.array([[0.9 * w, 0, 0.47 * w], [0, 0.9 * w, 0.52 * h], [0, 0, 1]])


@pytest.mark.parametrize("w,h,vs,shift", [(33, 9, 0.02, 0), (64, 16, 0.005, 0), (31, 7, 0.02, -3000), (70, 17, 0.05, 0.4),
                                          (33, 9, 0.0009, 0), (40, 11, 0.02, 25000), (40, 11, 0.02, -25000), (1, 1, 0.01, 0)])
def test_block_sets_match_oracle(w, h, vs, shift):
    K = K_of(w, h)
    vm = VoxelMapping(w, h, K, voxel_format="ref", with_color=False)
    vm.CreateMap(0, 1 << 16, vs)
    om = O.OracleMap(w, h, K, 1 << 16, vs, storage="ref")
    for seed in (1, 2):
        d, p = depth_and_pose(w, h, [shift, -0.5 * shift, 0.1 * shift], seed)
        vm.FuseDepth(to_gpu_depth(d), p)
        om.fuse(synth.depth_to_metres(d), None, p)
    st = vm.stats()
    assert st["error_flags"] == 0 and st["allocated_blocks"] == om.num_blocks() > 0
    assert set(block_keys(vm.export_blocks()["coords"]).tolist()) == set(block_keys(om.export()["coords"]).tolist())


def test_batch_that_mixes_near_and_far():
    import torch
    w, h = 40, 11
    K = K_of(w, h)
    cases = [(0.02, 0), (0.02, 25000), (0.0009, 0)]
    maps, want, frames = [], [], []
    for i, (vs, shift) in enumerate(cases):
        d, p = depth_and_pose(w, h, [shift, 0, 0], i)
        vm = VoxelMapping(w, h, K, voxel_format="f16", with_color=False)
        vm.CreateMap(0, 1 << 15, vs)
        om = O.OracleMap(w, h, K, 1 << 15, vs, storage="f16")
        om.fuse(synth.depth_to_metres(d), None, p)
        maps.append(vm)
        frames.append((to_gpu_depth(d), p))
        want.append(set(block_keys(om.export()["coords"]).tolist()))
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    b = MapBatch(maps)
    b.step([f[0] for f in frames], None, [f[1] for f in frames], [None] * 3, None, stream=s.cuda_stream)
    s.synchronize()
    for vm, k in zip(maps, want):
        assert set(block_keys(vm.export_blocks()["coords"]).tolist()) == k
