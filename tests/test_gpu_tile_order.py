"""The three orders of the ray marcher's tiles (0 bottom rows first, 1 top rows
first, 2 alternating from both ends) give the same images on a map and on both
schedules of a batch; maps and batches start with the alternating one."""
import numpy as np
import pytest
import torch

from voxelmapping_b200 import MapBatch, VoxelMapping, synth
from common import to_gpu_depth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]


def new_map(w, h):
    vm = VoxelMapping(w, h, WL.K, voxel_format="i16", with_color=False)
    vm.CreateMap(8, 1 << 14, 0.016)
    return vm


@pytest.mark.parametrize("w,h", [(33, 9), (161, 119)])
def test_orders_agree(w, h):
    d, _, pose = synth.Scene(WL).render(0)
    d = to_gpu_depth(np.ascontiguousarray(d[60:60 + h, 80:80 + w]))
    images = []
    for order in (0, 1, 2):
        vm = new_map(w, h)
        assert vm.get_launch_config()["raycast_tile_order"] == 2
        vm.set_launch_config(raycast_tile_order=order)
        assert vm.get_launch_config()["raycast_tile_order"] == order
        vm.FuseDepth(d, pose)
        images.append(vm.RenderScene(None, pose).cpu().numpy())
        for schedule in (1, 2):
            maps = [new_map(w, h), new_map(w, h)]
            b = MapBatch(maps)
            assert b.get_launch_config()["raycast_tile_order"] == 2
            b.set_launch_config(raycast_tile_order=order, batch_schedule=schedule)
            out = [torch.full((h, w, 4), float("nan"), device="cuda") for _ in maps]
            s = torch.cuda.Stream()
            torch.cuda.synchronize()
            b.step([d, d], None, [pose, pose], out, stream=s.cuda_stream)
            s.synchronize()
            images += [o.cpu().numpy() for o in out]
    assert np.isfinite(images[0]).any()
    assert all(np.array_equal(i, images[0], equal_nan=True) for i in images)
