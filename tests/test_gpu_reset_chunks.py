"""A reset zeroes every byte of the blocks in use, at counts around the chunks it
hands out (32 KB) from 120 MB on and the CTAs that take them, several times in a
row with different counts, and leaves no counter behind. The maps live in caller
memory."""
import ctypes as C

import numpy as np
import pytest
import torch

from voxelmapping_b200 import VoxelMapping
from voxelmapping_b200 import _lib as L

pytestmark = pytest.mark.gpu
K = np.array([[50.0, 0, 32], [0, 50.0, 24], [0, 0, 1]])


def up(n):
    return -(-n // 256) * 256


def fill(vm, n):
    """Load a snapshot of n blocks whose pool bytes are all non-zero."""
    i = np.arange(n)
    keys = (((i & 63) << 42) | ((i >> 6 & 63) << 21) | (i >> 12)).astype(np.uint64)
    h = L.SnapshotHeader.from_buffer_copy(vm.save_snapshot()[:64].tobytes())
    h.n_blocks = n
    h.pool_offset = up(h.keys_offset + keys.nbytes)
    snap = torch.full((h.pool_offset + n * h.block_bytes,), 0x3C, dtype=torch.uint8, device="cuda")
    snap[:C.sizeof(h)] = torch.from_numpy(np.frombuffer(bytes(h), np.uint8).copy()).cuda()
    snap[h.keys_offset:h.keys_offset + keys.nbytes] = torch.from_numpy(keys.view(np.uint8)).cuda()
    vm.load_snapshot(snap)
    return h.block_bytes


# blocks of 4,096 (f32), 5,632 (f32 + colour) and 2,048 bytes (ref): 8, 5.8 and 16 to a chunk; 8 CTAs on each of 148 SMs
EDGE = (120 << 20) // 2048  # ref blocks from which on the chunks are handed out


@pytest.mark.parametrize("fmt,color,counts", [("f32", False, [1, 8, 9]), ("f32", True, [6, 23000, 7000, 22345]),
                                              ("ref", False, [EDGE - 1, EDGE, EDGE + 1, EDGE + 15, 65536]), ("f32", False, [50001, 30721])])
def test_pool_is_zero_after_reset(fmt, color, counts):
    cap, buckets = 1 << 16, 1 << 16
    vm = VoxelMapping(64, 48, K, voxel_format=fmt, with_color=color, num_buckets=buckets)
    mem = torch.zeros(vm.required_bytes(8, cap, 0.01), dtype=torch.uint8, device="cuda")
    vm.CreateMapIn(8, cap, 0.01, mem)
    for n in counts:
        block = fill(vm, n)
        at = up(buckets * 4 * 16) + up(cap * 28) + up(cap * 8)
        pool, ctr = mem[at:at + cap * block], mem[at + up(cap * block):at + up(cap * block) + 64]
        assert vm.stats()["allocated_blocks"] == n and int(torch.count_nonzero(pool)) == n * block
        vm.reset()
        assert int(torch.count_nonzero(pool)) == 0 and int(torch.count_nonzero(ctr)) == 0
        assert vm.stats()["allocated_blocks"] == 0
