"""Treelet restructuring at the sizes where its treelets and their size classes change (3 to
8 leaves, a warp's and a block's worth of pieces), equal costs included, against the
oracle's restatement: the same topology words, boxes and triangles."""
import numpy as np
import pytest
import torch

import cpt
from cpt.device import DeviceLbvh, to_device
from oracle import cpu

pytestmark = pytest.mark.gpu


def records(lb, n, flags):
    lb.split(0.0, flags=flags)
    torch.cuda.synchronize()
    lb.status()
    return lb.split_nodes.cpu().numpy()[: (n - 1) * 96].view(np.float32).reshape(n - 1, 24).copy()


@pytest.mark.parametrize("copies", [1, 3])
@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 8, 9, 12, 31, 33, 129, 1000])
def test_treelet_sizes_match_oracle(cuda, n, copies):
    base = cpt.scene_random(max(n // copies, 2) + 4, seed=n, edge_min=0.05, edge_max=0.6)[0]
    tris = np.concatenate([base] * copies)[:n].copy()
    lb = DeviceLbvh(n, 63)
    lb.build(to_device(tris))
    rec0, rec1 = records(lb, n, 0), records(lb, n, cpt.SPLIT_TREELET)
    srt = lb.download()["tris"]
    lo = np.minimum(np.minimum(srt["v0"], srt["v1"]), srt["v2"])
    hi = np.maximum(np.maximum(srt["v0"], srt["v1"]), srt["v2"])
    words, right = rec0[:, 20].view(np.uint32), rec0[:, 21].view(np.uint32)
    leaf_boxes = np.zeros((n, 6), np.float32)
    for side in (0, 1):
        leaf = ((words >> side) & 1) == 0
        ids = ((words >> 2) if side == 0 else right)[leaf]
        tri = rec0[leaf, 10 * side + 3].view(np.uint32)
        leaf_boxes[ids] = np.concatenate([lo[tri], hi[tri]], 1)
    want = cpu.treelet(rec0, n, leaf_boxes, 4)
    assert np.array_equal(rec1[:, 20:24].view(np.uint32), want[:, 20:24].view(np.uint32))
    assert np.array_equal(rec1[:, :20], want[:, :20])
