"""Marching cubes by bit rows against the oracle where it can go wrong: block
faces, edges and corners (a surface through every neighbour), missing
neighbours, unobserved voxels, blocks with more triangles than a warp lists at
a time, an output buffer that ends inside a block, normals left out."""
import ctypes as C

import numpy as np
import pytest

from common import fuse_both, make_pair, sorted_rows
from voxelmapping_b200 import _lib as L
from voxelmapping_b200 import synth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]


def noisy_pair(fmt, vs, frames, noise, dropout):
    from dataclasses import replace
    w, h = 97, 73
    K = np.array([[80.0, 0, 48.0], [0, 80.0, 36.0], [0, 0, 1]])
    vm, om = make_pair(replace(WL, voxel_size=vs, num_blocks=1 << 14, num_entries=1 << 16), fmt=fmt, width=w, height=h, K=K)
    rng = np.random.default_rng(3)
    sc = synth.Scene(WL)
    for i in frames:
        d, _, pose = sc.render(i)
        d = d[::3, ::3][:h, :w].astype(np.int32)
        d = np.pad(d, ((0, 0), (0, 0))) + rng.integers(-noise, noise + 1, d.shape)
        d[rng.random(d.shape) < dropout] = 0
        full = np.zeros((h, w), np.uint16)
        full[:d.shape[0], :d.shape[1]] = np.clip(d, 0, 60000)
        fuse_both(vm, om, full, None, pose)
    return vm, om


def oracle_rows(om):
    n, v, nr = om.polygonize()[:3]
    return n, sorted_rows(np.concatenate([np.asarray(v, np.float32).reshape(n, 9), np.asarray(nr, np.float32).reshape(n, 9)], 1))


@pytest.mark.parametrize("fmt", ["ref", "f32", "f16", "i16"])
@pytest.mark.parametrize("vs,noise,dropout", [(0.05, 3, 0.02), (0.02, 60, 0.3)])
def test_triangles_match_oracle(fmt, vs, noise, dropout):
    vm, om = noisy_pair(fmt, vs, (0, 9, 50), noise, dropout)
    n, v, nr = vm.Polygonize()
    want, rows = oracle_rows(om)
    assert n == want > 1000
    assert np.array_equal(sorted_rows(np.concatenate([v, nr], 1)), rows)
    assert vm.stats()["last_triangles"] == n and vm.stats()["error_flags"] == 0


def test_crowded_blocks_and_short_buffers():
    import torch
    vm, om = noisy_pair("f32", 0.02, (0,), 0, 0.0)
    # random signs make most cubes cross the surface: up to 5 triangles each
    snap = vm.save_snapshot()
    h = L.SnapshotHeader.from_buffer_copy(snap[:C.sizeof(L.SnapshotHeader)].tobytes())
    words = snap[h.pool_offset:].reshape(h.n_blocks, h.block_bytes)[:, :4096].copy().view(np.float32).reshape(h.n_blocks, 512, 2)
    words[..., 0] = np.random.default_rng(1).uniform(-1, 1, words.shape[:2])
    words[..., 1] = 1.0
    new = snap.copy()
    new[h.pool_offset:].reshape(h.n_blocks, h.block_bytes)[:, :4096] = words.reshape(h.n_blocks, 1024).view(np.uint8)
    vm.load_snapshot(new)
    n, v, nr = vm.Polygonize()
    assert n > 600 * h.n_blocks  # more than one list per block
    rows = sorted_rows(np.concatenate([v, nr], 1))
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for cap in (n, n - 1, 1000, 33, 1):
        verts = torch.full((cap + 64, 9), -7.0, device="cuda")
        norms = torch.full((cap + 64, 9), -7.0, device="cuda")
        cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
        vm.clear_errors()
        for out in (norms, None):
            L.check(vm._lib.vmap_polygonize(vm._map, verts.data_ptr(), out.data_ptr() if out is not None else None, cap,
                                            cnt.data_ptr(), stream))
        assert int(cnt.item()) == n
        assert bool(vm.stats()["error_flags"] & L.FLAG_BUFFER_FULL) == (cap < n)
        assert bool((verts[cap:] == -7.0).all()) and bool((norms[cap:] == -7.0).all())
        got = verts[:cap].cpu().numpy()
        assert not (got == -7.0).any()
        if cap == n:
            assert np.array_equal(sorted_rows(got), sorted_rows(np.ascontiguousarray(rows[:, :9])))
