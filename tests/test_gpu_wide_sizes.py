"""The wide build at small sizes (a root alone, one and two levels, a warp's four groups, a
block's sixteen) and with equal areas and costs, both collapses: hits and occlusion are the
binary tree's, byte for byte but for exact ties."""
import numpy as np
import pytest
import torch

import cpt
from cpt.device import DeviceLbvh, to_device
from test_gpu_split import tie_or_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sah", [False, True])
@pytest.mark.parametrize("split", [0.0, 2.0])
@pytest.mark.parametrize("n", [2, 3, 4, 7, 8, 9, 15, 17, 33, 65, 129, 1025])
def test_wide_sizes(cuda, n, split, sah):
    tris = cpt.scene_random(n, seed=n, edge_min=0.1, edge_max=0.8)[0][:n].copy()
    tris[n // 2:]["v0"], tris[n // 2:]["v1"], tris[n // 2:]["v2"] = (tris[: n - n // 2][k] for k in ("v0", "v1", "v2"))
    lb = DeviceLbvh(n, 63)
    lb.build(to_device(tris))
    rng = np.random.default_rng(n)
    rays = np.zeros((3000, 8), np.float32)
    rays[:, :3] = rng.uniform(-1.0, 2.0, (3000, 3))
    rays[:, 4:7] = rng.uniform(0.0, 1.0, (3000, 3)) - rays[:, :3]
    d = torch.from_numpy(rays).cuda()
    want, _ = lb.trace(d)
    shade, _ = lb.trace(d, any_hit=True)
    if split:
        lb.split(split)
    lb.wide(sah=sah)
    got, _ = lb.trace(d)
    occluded, _ = lb.trace(d, any_hit=True)
    torch.cuda.synchronize()
    lb.status()
    ok, _ = tie_or_equal(got.cpu().numpy(), want.cpu().numpy())
    assert ok.all()
    assert torch.equal(occluded[:, 0] < 3e38, shade[:, 0] < 3e38)
    leaves = lb.bvh.split_capacity if split else n
    words = lb.status_words()
    assert 1 <= words[2] <= max(leaves - 1, 1) and n <= words[3] + 1
