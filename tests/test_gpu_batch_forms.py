"""A batch whose steps change between the kernels' forms (near or far views to
fuse, narrow or wide views to render, all four combinations, on both staging
buffers, on two streams) gives what its maps give alone; the graphs recorded
for one combination are not replayed for another."""
import itertools

import numpy as np
import pytest
import torch

from voxelmapping_b200 import MapBatch, VoxelMapping, synth
from common import block_keys, to_gpu_depth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]
W, H = 161, 119
K = np.array([[132.0, 0, 80.0], [0, 132.0, 59.0], [0, 0, 1]])


def new_map():
    vm = VoxelMapping(W, H, K, voxel_format="f32", with_color=False)
    vm.CreateMap(1 << 14, 1 << 12, 0.016)
    return vm


def frame(i, shift):
    d, _, p = synth.Scene(WL).render(i)
    p = p.copy()
    p[:3, 3] += shift
    return to_gpu_depth(np.pad(d[::2, ::2], ((0, 0), (0, 1)))[:H, :W]), p


def test_steps_that_change_form():
    # 16 mm voxels, 2^12 blocks: narrow to 1,032 m, near to 16.7 km; map 0 stays by the origin
    near, narrow_far, far = 0.0, 5000.0, 18000.0
    shifts = {"near narrow": near, "near wide": narrow_far, "far wide": far}
    frames = {k: frame(7, s) for k, s in shifts.items()}
    home = [frame(i, 0.0) for i in (0, 3)]
    order = list(itertools.chain(*itertools.permutations(["near narrow", "near wide", "far wide", "far narrow"], 3)))[:48]
    maps, alone = [new_map() for _ in range(4)], [new_map() for _ in range(4)]
    b = MapBatch(maps)
    assert all(m.stats()["error_flags"] == 0 for m in maps)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    out = [torch.full((H, W, 4), float("nan"), device="cuda") for _ in maps]
    torch.cuda.synchronize()
    where = {"near narrow": 1, "near wide": 2, "far wide": 3, "far narrow": 3}
    hits = 0
    for n, what in enumerate(order):
        if n == 24:
            torch.cuda.synchronize()
        s = streams[n // 24]
        d0, p0 = home[n % 2]
        k = where[what]
        d1, p1 = frames["far wide" if what == "far narrow" else what]
        render = what != "far narrow"  # a far frame fused but not rendered: the narrow marcher beside far_alloc
        depths, poses, vm = [d0, None, None, None], [p0] * 4, [out[0], None, None, None]
        depths[k], poses[k], vm[k] = d1, p1, out[k] if render else None
        b.step(depths, None, poses, vm, stream=s.cuda_stream)
        s.synchronize()
        alone[0].FuseDepth(d0, p0)
        alone[k].FuseDepth(d1, p1)
        assert torch.equal(torch.nan_to_num(out[0], -9.0), torch.nan_to_num(alone[0].RenderScene(None, p0), -9.0)), (n, what)
        if render:
            assert torch.equal(torch.nan_to_num(out[k], -9.0), torch.nan_to_num(alone[k].RenderScene(None, p1), -9.0)), (n, what)
            hits += int(torch.isfinite(out[k][..., 0]).sum())
    assert hits > 1000
    for a, m in zip(alone, maps):
        ea, em = a.export_blocks(), m.export_blocks()
        assert np.array_equal(np.sort(block_keys(ea["coords"])), np.sort(block_keys(em["coords"])))
        assert m.stats()["error_flags"] == 0
