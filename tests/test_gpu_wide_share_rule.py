"""How a launch over a wide tree shares its rays goes by the tree's leaves and the number of
rays; the hits do not. On both sides of each line of the rule they are those of the counting
traversal, which shares nothing, and so is a frame's image."""
import pytest
import torch

import cpt
from cpt.device import DeviceLbvh, DeviceRenderer, DeviceScene, make_params, to_device
from test_gpu_split import random_rays

pytestmark = pytest.mark.gpu


def built(n):
    tris, infos = cpt.scene_random(n, seed=7)
    lb = DeviceLbvh(n, 63)
    lb.build(to_device(tris[:n]))
    lb.wide()
    return lb, infos[:n]


@pytest.mark.parametrize("leaves", [2, 3, 511, 512, 513, 2_048, 2_049, 65_535, 65_536, 65_537])
def test_trace(cuda, leaves):
    lb, _ = built(leaves)
    few = torch.cuda.get_device_properties(0).multi_processor_count * 128
    for n in (1, 31, few - 1, few, few + 1, 8 * few + 1):
        rays = torch.from_numpy(random_rays(n, 3, inside=True)).cuda()
        alone, _ = lb.trace(rays, stats=True)
        shared, _ = lb.trace(rays)
        torch.cuda.synchronize()
        lb.status()
        assert torch.equal(alone.view(torch.int32), shared.view(torch.int32)), n


@pytest.mark.parametrize("leaves", [512, 513, 65_536, 65_537])
def test_image(cuda, leaves):
    lb, infos = built(leaves)
    sc = DeviceScene(infos)
    cam = cpt.camera_look_at((0.5, 0.5, -1.2), (0.5, 0.5, 0.0), aspect=1.0)
    out = []
    for stats in (True, False):
        r = DeviceRenderer(make_params(150, 150, 1, 0, 3, 3.0, True, 9, trace_stats=stats))
        r.render(lb, sc, cam)
        torch.cuda.synchronize()
        r.check_status()
        out.append(r.accum.cpu().numpy().tobytes())
    assert out[0] == out[1]
