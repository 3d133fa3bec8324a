"""Builds whose launches start while the one before drains: many in a row on one stream, each on
other triangles and in the same buffers, and the same captured in a graph, against the oracle."""
import numpy as np
import pytest
import torch

import cpt
from cpt.device import DeviceLbvh, to_device
from oracle import cpu

pytestmark = pytest.mark.gpu

FIELDS = ("keys", "tris", "children", "parents_internal", "node_boxes")


def _same(out, ref):
    for f in FIELDS:
        assert np.ascontiguousarray(out[f]).tobytes() == np.ascontiguousarray(getattr(ref, f)).tobytes(), f


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [2, 257, 1025, 20_001, 98_305])
def test_builds_in_a_row(cuda, n, bits):
    hosts = [cpt.scene_random(n, seed=s)[0][:n].copy() for s in range(4)]
    devs = [to_device(t) for t in hosts]
    lb = DeviceLbvh(n, bits)
    torch.cuda.synchronize()
    for last in (3, 1):
        for d in devs + [devs[last]]:  # no synchronisation between them
            lb.build(d)
        torch.cuda.synchronize()
        lb.status()
        _same(lb.download(), cpu.build(hosts[last], bits))


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [257, 20_001])
def test_builds_in_a_graph(cuda, n, bits):
    hosts = [cpt.scene_random(n, seed=s)[0][:n].copy() for s in range(3)]
    devs = [to_device(t) for t in hosts]
    tris = devs[0].clone()
    lb = DeviceLbvh(n, bits)
    lb.build(tris)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        lb.build(tris)
        lb.build(tris)
    for i in (1, 2, 0):
        tris.copy_(devs[i])
        graph.replay()
        torch.cuda.synchronize()
        lb.status()
        _same(lb.download(), cpu.build(hosts[i], bits))
