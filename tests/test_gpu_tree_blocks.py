"""The tree over blocks of 256 leaves at the sizes where it changes (a block short of full,
full, one leaf over; two blocks; many), on key sequences that make deep and lopsided trees:
every array against the oracle, byte for byte, for single, batched and split builds."""
import numpy as np
import pytest
import torch

import cpt
from cpt.device import DeviceLbvh, LbvhBatch, to_device
from oracle import cpu

pytestmark = pytest.mark.gpu
FIELDS = ("keys", "tris", "children", "parents_leaf", "parents_internal", "node_boxes")


def soup(kind, n):
    t = cpt.scene_random(max(n, 2), seed=n + 1)[0][:n].copy()
    if kind == "equal":  # a handful of distinct keys: ties decided by position
        for v in ("v0", "v1", "v2"):
            t[v] = t[v][np.arange(n) % 5]
    elif kind == "spiral":  # every leaf splits from all that follow: as deep as keys allow
        x = 2.0 ** -np.linspace(0.0, 20.0, n)
        for v in ("v0", "v1", "v2"):
            t[v] = t[v] * 1e-7 + x[:, None].astype(np.float32)
    elif kind == "zeros":  # bounds that are zeros of both signs
        for v in ("v0", "v1", "v2"):
            t[v][:, 1] = np.where(np.arange(n) % 3 == 0, np.float32(-0.0), np.float32(0.0))
            t[v][:, 2] = np.abs(t[v][:, 2]) * np.where(np.arange(n) % 2 == 0, 1.0, 0.0)
    return t


def same(lb, tris, bits, box):
    ref, out = cpu.build(tris, bits, box=box) if box is not None else cpu.build(tris, bits), lb.download()
    for f in FIELDS:
        assert np.ascontiguousarray(out[f]).tobytes() == np.ascontiguousarray(getattr(ref, f)).tobytes(), f


@pytest.mark.parametrize("kind", ["random", "equal", "spiral", "zeros"])
@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [2, 3, 255, 256, 257, 511, 512, 513, 3000])
def test_tree_block_edges(cuda, n, bits, kind):
    tris = soup(kind, n)
    lb = DeviceLbvh(n, bits)
    lb.build(to_device(tris))
    torch.cuda.synchronize()
    lb.status()
    same(lb, tris, bits, None)


def test_batch_of_block_edges(cuda):
    sizes = (257, 2, 256, 1000, 255, 513)
    soups = [soup("equal" if i % 2 else "random", n) for i, n in enumerate(sizes)]
    lbs = [DeviceLbvh(n, 63) for n in sizes]
    LbvhBatch(lbs).build([to_device(t) for t in soups], np.stack([cpt.scene_bounds(t) for t in soups]))
    torch.cuda.synchronize()
    for lb, t in zip(lbs, soups):
        lb.status()
        one = DeviceLbvh(lb.n, 63)
        one.build(to_device(t), box=cpt.scene_bounds(t))
        torch.cuda.synchronize()
        a, b = lb.download(), one.download()
        for f in a:
            assert a[f].tobytes() == b[f].tobytes(), f


@pytest.mark.parametrize("n", [2, 90, 256, 300])
@pytest.mark.parametrize("ratio", [0.0, 3.0])
def test_split_tree_block_edges(cuda, n, ratio):
    """The split tree reaches every node and piece once, and the records past it are marked."""
    tris = soup("random", n)
    lb = DeviceLbvh(n, 63)
    lb.build(to_device(tris))
    lb.split(ratio)
    torch.cuda.synchronize()
    lb.status()
    cap = lb.bvh.split_capacity
    rec = lb.split_nodes.cpu().numpy()[: (cap - 1) * 96].view(np.uint32).reshape(cap - 1, 24)
    seen, leaves, stack = set(), [], [0]
    while stack:
        i = stack.pop()
        assert i not in seen
        seen.add(i)
        word, right = int(rec[i, 20]), int(rec[i, 21])
        for side, child in ((0, word >> 2), (1, right)):
            if (word >> side) & 1:
                stack.append(child)
            else:
                leaves.append(child)
                assert rec[i, 10 * side + 3] < n
    assert sorted(leaves) == list(range(len(leaves))) and len(leaves) == len(seen) + 1
    assert all(rec[i, 20] == 0xFFFFFFFF for i in range(cap - 1) if i not in seen)
