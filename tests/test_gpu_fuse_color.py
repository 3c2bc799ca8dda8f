"""Colour of a batch's fusion, read in two loads per pixel, against the oracle,
bit for bit: images at odd and even addresses, rows at odd and even pitches, the
last pixel at the end of its buffer, both depth types."""
import numpy as np
import pytest

from common import aligned_maps, make_pair
from voxelmapping_b200 import MapBatch, synth

pytestmark = pytest.mark.gpu
WL = synth.WORKLOADS["room_small"]


@pytest.mark.parametrize("fmt,float_depth", [("ref", False), ("f32", True), ("f16", False), ("i16", True)])
def test_batch_colour_at_any_alignment_matches_oracle(fmt, float_depth):
    import torch
    w, h = 157, 101
    K = np.array([[131.3, 0, 77.7], [0, 129.1, 51.2], [0, 0, 1]])
    places = [(0, 0), (1, 0), (0, 1), (3, 2)]  # bytes before the image, between its rows
    pairs = [make_pair(WL, fmt=fmt, color=True, width=w, height=h, K=K) for _ in places]
    batch = MapBatch([vm for vm, _ in pairs])
    sc = synth.Scene(WL)
    for i in (0, 7, 31):
        d, c, pose = sc.render(i)
        d, c = np.ascontiguousarray(d[::2, ::2][:h, :w]), np.ascontiguousarray(c[::2, ::2][:h, :w])
        m = synth.depth_to_metres(d, 0.001).astype(np.float32)
        depths = [torch.from_numpy(m).cuda() if float_depth else torch.from_numpy(d.view(np.int16)).cuda() for _ in places]
        rgbs = []
        for before, gap in places:
            buf = torch.zeros(before + h * (3 * w + gap) - gap, dtype=torch.uint8, device="cuda")
            rgb = torch.as_strided(buf, (h, 3 * w), (3 * w + gap, 1), before)
            rgb.copy_(torch.from_numpy(c.reshape(h, -1)))
            rgbs.append(rgb)
        batch.step(depths, rgbs, [pose] * len(places), [None] * len(places), [None] * len(places))
        torch.cuda.synchronize()
        for _, om in pairs:
            om.fuse(m, c, pose)
    for vm, om in pairs:
        g, o = aligned_maps(vm, om)
        assert np.array_equal(g["coords"], o["coords"]) and g["weight"].max() >= 2 and g["rgb"].max() > 0
        for k in ("tsdf", "weight", "rgb"):
            assert np.array_equal(g[k], o[k].astype(g[k].dtype)), k
    batch.release()
