"""Both forms of the fusion's projection against the FP32 oracle, bit for bit:
voxels around the camera plane (rows that cross it take the plain form, their
neighbours the packed one), voxels too large for the packed form at all, odd
image sizes, every format, with and without colour, three updates per voxel."""
import numpy as np
import pytest

from common import aligned_maps, fuse_both, make_pair
from voxelmapping_b200 import synth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]


@pytest.mark.parametrize("vs", [0.013, 0.25, 0.5, 1.5])
@pytest.mark.parametrize("fmt,color", [("ref", True), ("f32", True), ("f16", False), ("i16", True)])
def test_projection_forms_match_oracle(vs, fmt, color):
    from dataclasses import replace
    w, h = 157, 101
    K = np.array([[131.3, 0, 77.7], [0, 129.1, 51.2], [0, 0, 1]])
    wl = replace(WL, voxel_size=vs, num_blocks=1 << 14, num_entries=1 << 16)
    vm, om = make_pair(wl, fmt=fmt, color=color, width=w, height=h, K=K)
    sc = synth.Scene(WL)
    for i in (0, 7, 7, 31):
        d, c, pose = sc.render(i)
        d, c = np.ascontiguousarray(d[::2, ::2][:h, :w]), np.ascontiguousarray(c[::2, ::2][:h, :w])
        if vs > 1:  # blocks of 12 m are seen where a corner is: look down on the one at the origin
            pose = np.array([[1.0, 0, 0, 0.3], [0, -1, 0, 0.2], [0, 0, -1, 1.5], [0, 0, 0, 1]])
            d = np.full((h, w), 1490 + 5 * i, np.uint16)
        st, orc = fuse_both(vm, om, d, c if color else None, pose)
        assert st["visible_blocks"] == orc["visible"] and st["error_flags"] == 0
    g, o = aligned_maps(vm, om)
    assert np.array_equal(g["coords"], o["coords"])
    assert np.array_equal(g["weight"], o["weight"].astype(np.float32)) and g["weight"].max() >= 2
    assert np.array_equal(g["tsdf"], o["tsdf"].astype(np.float32))
    if color:
        assert np.array_equal(g["rgb"], o["rgb"])
