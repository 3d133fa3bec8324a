"""The end of a wide-tree traversal launch, where a warp's idle lanes take over parts of
the rays still under way: every ray's closest hit is the one that a lane finds alone
(the counting traversal, which shares nothing), whatever the number of rays, and so are
an image's bytes and shadow rays' visibility."""
import numpy as np
import pytest
import torch

import cpt
from cpt.device import BatchRenderer, DeviceLbvh, DeviceRenderer, DeviceScene, make_params, to_device
from oracle import cpu
from test_gpu_split import hairball, random_rays

pytestmark = pytest.mark.gpu


def built(tris, split=0.0, wide=True):
    lb = DeviceLbvh(len(tris), 63)
    lb.build(to_device(tris))
    if split:
        lb.split(split)
    if wide:
        lb.wide()
    return lb


# around a warp, the helped lanes of a warp (8), the threshold (12), a block; a grid with
# fewer rays than lanes, and one with more than a ray for every lane of the chip
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 12, 13, 31, 32, 33, 127, 129, 4097, 60_001, 400_003])
def test_hits_do_not_depend_on_helpers(cuda, n):
    tris, _ = hairball(n_hair=60_000)
    lb = built(tris, 1.25)
    rays = np.concatenate([random_rays(n - n // 2, 5), random_rays(n // 2, 6, inside=True)]) if n > 1 else random_rays(1, 5)
    d = torch.from_numpy(rays).cuda()
    alone, _ = lb.trace(d, stats=True)
    helped, _ = lb.trace(d)
    torch.cuda.synchronize()
    lb.status()
    assert helped.cpu().numpy().tobytes() == alone.cpu().numpy().tobytes()


@pytest.mark.parametrize("n", [40, 5_000])
def test_exact_ties_keep_the_visiting_order(cuda, n):
    """Every triangle three times over: each hit is a three-way tie, of which the traversal
    of one lane reports the first it visits."""
    base, _ = hairball(n_hair=4_000, nu=24, nv=12)
    tris = np.concatenate([base, base, base])
    for split in (0.0, 2.0):
        lb = built(tris, split)
        d = torch.from_numpy(random_rays(n, 11, inside=True)).cuda()
        alone, _ = lb.trace(d, stats=True)
        helped, _ = lb.trace(d)
        torch.cuda.synchronize()
        lb.status()
        assert helped.cpu().numpy().tobytes() == alone.cpu().numpy().tobytes()


def test_two_triangles_and_zero_directions(cuda):
    """The smallest tree (nothing to give away), and rays along the axes."""
    tris, _ = cpt.scene_random(2, seed=4)
    lb = built(tris[:2])
    rays = random_rays(300, 3)
    rays[::3, 4:7] = [0.0, 0.0, 1.0]
    rays[1::3, 4:7] = [-0.0, -1.0, 0.0]
    d = torch.from_numpy(rays).cuda()
    a, _ = lb.trace(d, stats=True)
    b, _ = lb.trace(d)
    torch.cuda.synchronize()
    assert a.cpu().numpy().tobytes() == b.cpu().numpy().tobytes()


@pytest.mark.parametrize("size", [(3, 2), (40, 30), (257, 129)])
def test_image_does_not_depend_on_helpers(cuda, size):
    tris, infos = hairball(n_hair=30_000)
    lb, sc = built(tris, 1.25), DeviceScene(infos)
    w, h = size
    cam = cpt.camera_look_at((0.0, 0.35, -3.6), (0.0, 0.0, 0.0), aspect=w / h)
    out = []
    for stats in (True, False):
        r = DeviceRenderer(make_params(w, h, 2, 0, 5, 3.0, True, 9, trace_stats=stats))
        r.render(lb, sc, cam)
        torch.cuda.synchronize()
        r.check_status()
        out.append((r.accum.cpu().numpy().tobytes(), r.counts[:3].cpu().numpy().tolist()))
    assert out[0] == out[1]


@pytest.mark.parametrize("size", [(3, 2), (64, 48)])
def test_shadow_rays_against_the_oracle(cuda, size):
    """Next-event estimation over the wide tree, whose shadow rays are shared among lanes
    too, against the oracle (random triangles: no ray is lost by its box test)."""
    tris, infos = cpt.scene_random(20_000, seed=5)
    w, h = size
    lb, sc = built(tris), DeviceScene(infos)
    sc.build_emitters(lb, 1 << 14)
    cam = cpt.camera_look_at((0.5, 0.5, -1.2), (0.5, 0.5, 0.0), aspect=w / h)
    r = DeviceRenderer(make_params(w, h, 4, 5, 3, 3.0, True, 77, nee=True))
    r.render(lb, sc, cam)
    torch.cuda.synchronize()
    r.check_status()
    b = cpu.build(tris, 63)
    table, _ = cpu.emitters(b, infos, 1 << 14)
    ocam = cpu.ocam_from(cam.eye, cam.as_array()[3:], np.ctypeslib.as_array(cam.inv_view_proj))
    rad, counts = cpu.render(b, infos, None, w, h, 4, 5, 3, 3.0, True, 77, ocam, nee_table=table)
    s, _, _ = cpu.accumulate_kahan(rad)
    assert r.accum.cpu().numpy().view(np.float32).reshape(2, h, w, 4)[0][..., :3].tobytes() == s.tobytes()
    assert np.array_equal(r.counts.cpu().numpy()[:3].astype(np.uint64), counts)


def test_views_of_several_scenes(cuda):
    """Rays of different trees in one warp: a helper takes over its donor's tree with the ray."""
    specs = [(hairball(n_hair=9_000, seed=s), s) for s in (1, 2, 3)]
    params = make_params(0, 0, 1, 0, 4, 3.0, True, 5)
    cam = cpt.camera_look_at((0.0, 0.35, -3.6), (0.0, 0.0, 0.0), aspect=1.0)
    views = [(built(t), DeviceScene(i), cam, 24, 24) for (t, i), _ in specs]
    both = BatchRenderer(views, params)
    both.render()
    stats = BatchRenderer(views, make_params(0, 0, 1, 0, 4, 3.0, True, 5, trace_stats=True))
    stats.render()
    torch.cuda.synchronize()
    both.check_status()
    for a, b in zip(both.accums, stats.accums):
        assert a.cpu().numpy().tobytes() == b.cpu().numpy().tobytes()
