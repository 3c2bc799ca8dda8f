"""The ray marcher's narrow form (floors by one add, whole empty cubes crossed
without lookups) renders, bit for bit, what its wide form renders of the same
map: a batch's persistent step always marches wide, a map's own call narrow
while the view is within 2,080 m here. Ordinary views of a room at the origin and
shifted along every axis, both raycast modes, every storage format."""
import numpy as np
import pytest
import torch

from voxelmapping_b200 import MapBatch, VoxelMapping, synth
from common import to_gpu_depth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]
W, H = 161, 119
K = np.array([[132.0, 0, 80.0], [0, 132.0, 59.0], [0, 0, 1]])


@pytest.mark.parametrize("fmt,mode", [("f32", 0), ("f32", 1), ("ref", 0), ("f16", 1), ("i16", 0)])
@pytest.mark.parametrize("shift", [(0, 0, 0), (-900, 450, 30), (3, -1700, -800), (25, 60, 1900)])
def test_forms_agree(fmt, mode, shift):
    sc = synth.Scene(WL)
    vm = VoxelMapping(W, H, K, voxel_format=fmt, with_color=False, raycast_mode=mode)
    vm.CreateMap(1 << 17, 1 << 15, 0.016)  # 32 cells on the shortest axis
    poses = []
    for i in (0, 12, 24, 60):
        d, _, p = sc.render(i)
        p = p.copy()
        p[:3, 3] += shift
        poses.append(p)
        if i < 60:
            vm.FuseDepth(to_gpu_depth(np.pad(d[::2, ::2], ((0, 0), (0, 1)))[:H, :W]), p)
    b = MapBatch([vm])
    b.set_launch_config(batch_schedule=2)
    s = torch.cuda.Stream()
    hits = 0
    for p in poses:
        wide = torch.full((H, W, 4), float("nan"), device="cuda")
        narrow = vm.RenderScene(None, p)
        torch.cuda.synchronize()
        b.step([None], None, [p], [wide], stream=s.cuda_stream)
        s.synchronize()
        a, c = narrow.cpu().numpy(), wide.cpu().numpy()
        assert np.array_equal(a, c, equal_nan=True), int((a != c).any(-1).sum())
        hits += int(np.isfinite(a[..., 0]).sum())
    assert hits > 10000 and vm.stats()["error_flags"] == 0
    b.release()
