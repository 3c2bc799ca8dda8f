"""Rays almost parallel to a face of a large empty cube: the jumps over the cube's
blocks that are taken without a lookup must not carry a ray past a block of the
neighbouring cube. The map is a wall one block wide beside the face, loaded from
a snapshot; the narrow form of the ray marcher, which crosses whole empty cubes,
is compared with the wide form, which looks every block up (a map whose few
buckets leave no room for a block grid)."""
import ctypes as C

import numpy as np
import pytest

from voxelmapping_b200 import VoxelMapping
from voxelmapping_b200 import _lib as L

pytestmark = pytest.mark.gpu
W, H, VS = 64, 32, 0.02


def new_map(f, blocks, buckets, mode):
    K = np.array([[f, 0, 31.37], [0, f, 15.73], [0, 0, 1]])
    vm = VoxelMapping(W, H, K, voxel_format="f32", with_color=False, num_buckets=buckets, raycast_mode=mode)
    vm.CreateMap(8, blocks, VS)
    return vm


def snapshot(vm, blocks, tsdf):
    """A snapshot of `blocks` (n, 3), every voxel of weight 1 and TSDF tsdf(n, 512)."""
    keys = np.zeros(len(blocks), np.uint64)
    for a in range(3):
        keys = keys << np.uint64(21) | (np.asarray(blocks)[:, a].astype(np.int64) & 0x1FFFFF).astype(np.uint64)
    h = L.SnapshotHeader.from_buffer_copy(vm.save_snapshot()[:64].tobytes())
    h.n_blocks = len(blocks)
    h.pool_offset = (h.keys_offset + keys.nbytes + 255) // 256 * 256
    pool = np.stack([tsdf, np.ones_like(tsdf)], -1).astype(np.float32)
    out = np.zeros(h.pool_offset + pool.nbytes, np.uint8)
    out[:C.sizeof(h)] = np.frombuffer(bytes(h), np.uint8)
    out[h.keys_offset:h.keys_offset + keys.nbytes] = keys.view(np.uint8)
    out[h.pool_offset:] = pool.reshape(-1).view(np.uint8)
    return out


def wall(axis, face, sign, near, side):
    """Blocks of the wall and their TSDF: along `axis` the column of blocks next to the face at voxel `face`, on the side
    that rays drifting in direction `sign` come to; along z the two blocks about the surface, 104 voxels past `near`."""
    other = 1 - axis
    blocks, tsdf = [], []
    z = np.arange(8)[:, None, None]
    for bz in range((near + 96) // 8, (near + 112) // 8):
        for o in range(side // 8 - 2, side // 8 + 2):
            b = [0, 0, bz]
            b[axis] = face // 8 if sign > 0 else face // 8 - 1
            b[other] = o
            blocks.append(b)
            tsdf.append(np.broadcast_to(np.clip((near + 104.25 - (bz * 8 + z)) / 4, -1, 1), (8, 8, 8)).reshape(512))
    return np.array(blocks), np.array(tsdf)


# the face's distance from the origin in voxels; the larger it is, the coarser the positions' floats
@pytest.mark.parametrize("face", [1024, 3968, -16000, 32000])
@pytest.mark.parametrize("axis", [0, 1])
# rays that drift down see the wall only a voxel past the face (its reads need the next voxel up): steeper ones alone
@pytest.mark.parametrize("sign,f", [(1, 5.0e2), (1, 2.0e4), (1, 2.0e5), (-1, 5.0e2)])
def test_rays_beside_a_cube_face(face, axis, sign, f):
    near, side = 256, 2048 + 64
    narrow, wide = new_map(f, 1 << 12, 0, 1), new_map(f, 32, 9, 1)
    blocks, tsdf = wall(axis, face, sign, near, side)
    for vm in (narrow, wide):
        vm.load_snapshot(snapshot(vm, blocks, tsdf))
    hits = 0
    for step in range(24):
        # the rays of column (row) step + 0.5 past the image centre reach the face where the surface is
        p = np.eye(4)
        p[axis, 3] = (face - sign * (step + 0.5) / f * 104) * VS
        p[1 - axis, 3] = (side + 0.3) * VS
        p[2, 3] = (near + 0.1) * VS
        a, b = (vm.RenderScene(None, p).cpu().numpy() for vm in (narrow, wide))
        assert np.array_equal(a, b, equal_nan=True), (step, int((np.isfinite(a) != np.isfinite(b)).any(-1).sum()))
        hits += int(np.isfinite(b[..., 0]).sum())
    assert hits > 1000
