"""The radix sort at its tile sizes' edges (1,024 keys up to 98,304 elements, 2,048 up to
786,432, then 4,096; a tile short, full and one over): a build's keys, order and tree against
the oracle, both key widths, and the static build's scratch at each."""
import numpy as np
import pytest
import torch

import cpt
from cpt.device import DeviceLbvh, stream_handle, to_device
from oracle import cpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [30, 63])
@pytest.mark.parametrize("n", [1023, 1024, 1025, 98_303, 98_304, 98_305, 100_353, 786_431, 786_432, 786_433, 790_529])
def test_tile_edges(cuda, n, bits):
    tris = cpt.scene_random(n, seed=n)[0][:n].copy()
    tris[::3] = tris[0]  # many equal keys: the order among them is the input's
    tris["info_idx"] = np.arange(n, dtype=np.uint32)
    lb = DeviceLbvh(n, bits)
    lb.build(to_device(tris))
    torch.cuda.synchronize()
    lb.status()
    ref, out = cpu.build(tris, bits), lb.download()
    for f in ("keys", "tris", "children", "parents_internal", "node_boxes"):
        assert np.ascontiguousarray(out[f]).tobytes() == np.ascontiguousarray(getattr(ref, f)).tobytes(), f


@pytest.mark.parametrize("n", [2, 98_304, 98_305, 131_072])
def test_static_build_at_tile_edges(cuda, n):
    tris = cpt.scene_random(n, seed=n)[0][:n].copy()
    lb = DeviceLbvh(n, 63)
    d = to_device(tris)
    cpt.check(cpt.lib.cpt_lbvh_build_static(d.data_ptr(), n, None, 63, cpt.device.ctypes.byref(lb.bvh), 0,
                                            stream_handle()), "cpt_lbvh_build_static")
    torch.cuda.synchronize()
    lb.status()
    ref, out = cpu.build(tris, 63), lb.download()
    assert out["keys"].tobytes() == ref.keys.tobytes() and out["children"].tobytes() == ref.children.tobytes()


def test_scratch_sizes_grow_with_the_count(cuda):
    """Scratch sized for one count serves every smaller one, across the tile sizes' edges."""
    counts = [2, 1024, 50_000, 98_303, 98_304, 98_305, 98_400, 110_000, 131_072, 400_000, 786_431, 786_432, 786_433,
              800_000, 1_000_000, 2_000_000]
    for bits in (30, 63):
        single = [cpt.lbvh_scratch_bytes(n, bits) for n in counts]
        batch = [cpt.lib.cpt_lbvh_batch_scratch_bytes((cpt.device.ctypes.c_uint32 * 1)(n), 1, bits) for n in counts]
        split = [cpt.lib.cpt_lbvh_split_bytes(n, bits, 0.0, 0, None) for n in counts]
        for sizes in (single, batch, split):
            assert sizes == sorted(sizes) and all(sizes)
    assert cpt.lbvh_scratch_bytes(131_072, 63) <= 8 << 20
