"""Triangles with NaN coordinates: min and max that select their second argument are not
associative over NaN, so the boxes show in which order they were united. They are the
reference order's (child by child up the tree, the oracle's), in one block of leaves and
across blocks, for single and batched builds."""
import numpy as np
import pytest
import torch

import cpt
from cpt.device import DeviceLbvh, LbvhBatch, to_device
from oracle import cpu

pytestmark = pytest.mark.gpu

ARRAYS = ("keys", "tris", "children", "parents_leaf", "parents_internal", "node_boxes")
BOX = np.array([0, 0, 0, 1, 1, 1], np.float32)


def with_nans(n, seed, every):
    tris = cpt.scene_random(n, seed=seed)[0].copy()
    g = np.random.default_rng(seed)
    for i in g.choice(len(tris), max(1, len(tris) // every), replace=False):
        tris[("v0", "v1", "v2")[g.integers(0, 3)]][i, g.integers(0, 3)] = np.nan
    return tris


def same(lb, tris, bits):
    out, ref = lb.download(), cpu.build(tris, bits, BOX)
    for k in ARRAYS:
        assert np.ascontiguousarray(out[k]).tobytes() == np.ascontiguousarray(getattr(ref, k)).tobytes(), k


# a block of leaves is 256: the tree inside one, on its edge, across two and many
@pytest.mark.parametrize("n", [3, 64, 254, 255, 512, 3000, 60_000])
@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("every", [3, 50])
def test_boxes_are_united_in_tree_order(cuda, n, bits, every):
    tris = with_nans(n, n, every)
    lb = DeviceLbvh(len(tris), bits)
    lb.build(to_device(tris), box=BOX)
    torch.cuda.synchronize()
    same(lb, tris, bits)


def test_batched(cuda):
    scenes = [with_nans(n, n, 10) for n in (40, 300, 5000)]
    lbs = [DeviceLbvh(len(t), 63) for t in scenes]
    LbvhBatch(lbs).build([to_device(t) for t in scenes], np.stack([BOX] * 3))
    torch.cuda.synchronize()
    for lb, t in zip(lbs, scenes):
        same(lb, t, 63)
