"""Triangles a thousand times as far as the rays reach: their coordinates round
by more than anything near the camera, so whether a ray grazes one is decided
by the rounding of the triangle test itself, and the packets' cull before it
may not decide otherwise. The triangles below are ones whose vertices the
frustum's plane has all on its outer side, as FP32 evaluates it, while the
triangle test reports a hit (found by evaluating both on the CPU)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import T, gpu_forward, settings  # noqa: E402

GRAZED = np.array([
    1141798.0, -789913.4375, 2487463.25, -1214383.625, 839958.25, -2645588.25, -0.6809107065200806, 2200.148193359375, 1.534092664718628,
    -1355986.25, -294711.53125, 3798105.25, 614696.0625, 133522.5625, -1721753.875, 1.4696683883666992, 771.8721313476562, -1.1469353437423706,
    -291074.5625, 553263.5, 815299.5625, 328655.90625, -623787.9375, -920558.5625, 1.5621830224990845, -453.8656311035156, -1.399655818939209,
    500413.0, 3303507.25, 1090176.125, -1089189.875, -7183648.0, -2372848.0, -0.9548452496528625, -57998.3828125, 0.9387833476066589,
    -570076.8125, 2904789.0, 1596781.625, 1183333.25, -6024657.5, -3314500.0, 0.7134801745414734, -3163.497802734375, 0.9713900685310364,
    -1579279.375, 2224589.0, 3440537.0, 1674555.25, -2358336.5, -3648093.75, 1.3380106687545776, -3068.506103515625, 0.10758212208747864,
    -333305.625, 2127480.5, 933588.3125, 1384012.25, -8825803.0, -3876600.0, 1.036402940750122, -49215.9140625, 0.06745914369821548,
    425949.84375, -1051772.25, 1193083.625, -884812.125, 2184054.0, -2478345.75, -1.758501410484314, 930.5297241210938, -1.9538723230361938,
], np.float32).reshape(-1, 3, 3)


def _hits(tr, tri, ro, rd):
    """Hits the passes evaluated, over all rays."""
    sc = scenes.make_scene(1, seed=3)
    sc.verts[:] = tri
    tr.reset_stats()
    gpu_forward(tr, sc, ro, rd, settings())
    tr.device_status()
    return tr.stats()["evaluated_hits"]


@pytest.mark.parametrize("copies", [1, 16], ids=["rays", "tiles"])
def test_grazed_triangles_are_not_culled(copies):
    # 16 copies of the image: more tiles than half the warps, so a warp has a whole one
    ro, rd = (np.tile(a, (copies, 1, 1)) for a in scenes.camera_rays(scenes.look_at_camera([0.0, 0.0, 3.0], 64, 64)))
    tr = _C.OptixTracer()
    tr.set_traversal("lanes", 16, 32)
    want = [_hits(tr, tri, ro, rd) for tri in GRAZED]
    assert min(want) >= copies
    for k in (16, 32):
        tr.set_traversal("packets", k)
        assert [_hits(tr, tri, ro, rd) for tri in GRAZED] == want
