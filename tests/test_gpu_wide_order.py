"""Thin triangles from far away: the distance computed for a hit may lie before the box that
holds the triangle, so a hit can hang on the order in which boxes are visited. A launch that
shares its last rays among lanes reports the hits of one lane alone (the counting traversal,
which shares nothing), in every run and whatever rays share a warp."""
import numpy as np
import pytest
import torch

from cpt.device import DeviceLbvh, to_device
from test_gpu_split import hairball

pytestmark = pytest.mark.gpu


def rays_from(distance, n, seed):
    g = np.random.default_rng(seed)
    d0 = g.normal(size=(n, 3))
    o = distance * d0 / np.linalg.norm(d0, axis=1, keepdims=True)
    d = g.uniform(-1.0, 1.0, (n, 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = o
    r[:, 4:7] = d
    return r


@pytest.mark.parametrize("split", [0.0, 2.0])
@pytest.mark.parametrize("distance", [20.0, 100.0, 400.0])
def test_far_hits_do_not_depend_on_the_order(cuda, distance, split):
    tris, _ = hairball(n_hair=400_000)
    lb = DeviceLbvh(len(tris), 63)
    lb.build(to_device(tris))
    if split:
        lb.split(split)
    lb.wide()
    rays = torch.from_numpy(rays_from(distance, 20_000, 7)).cuda()
    alone, _ = lb.trace(rays, stats=True)
    for run in range(4):
        order = torch.randperm(len(rays), device="cuda") if run % 2 else torch.arange(len(rays), device="cuda")
        helped, _ = lb.trace(rays[order].contiguous())
        torch.cuda.synchronize()
        lb.status()
        assert helped.cpu().numpy().tobytes() == alone[order].cpu().numpy().tobytes(), run
