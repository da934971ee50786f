"""The sphere programs trace their rays as pairs or one a lane, by the image's
size, the tree's and the hits to expect: on both sides of the rule's lines the
images are the same, bit for bit, as those of the image's parts, which are too
small for a ray a lane."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import gpu_forward, settings  # noqa: E402
from scenes_for_tests import sphere_extra  # noqa: E402

SCENES = {
    "small": lambda: scenes.make_scene(1000, seed=1),  # a ray a lane above 141k pixels
    "large": lambda: scenes.make_scene(60_000, seed=2),  # above 731k
    "dense": lambda: scenes.make_scene(3000, seed=3, center_std=0.15, edge_range=(0.05, 0.3)),  # never
    "one": lambda: scenes.make_scene(1, seed=7, center_std=0.01, edge_range=(0.3, 0.5)),
}


@pytest.mark.parametrize("program,samples", [("reflect.ptx", 0), ("refract.ptx", 0), ("envlight.ptx", 1)])
@pytest.mark.parametrize("scene,h,w", [("small", 361, 401), ("small", 353, 400), ("large", 850, 870), ("dense", 400, 400),
                                       ("one", 365, 400)])
def test_image_equals_its_parts(scene, h, w, program, samples):
    sc = SCENES[scene]()
    ro, rd = scenes.camera_rays(scenes.look_at_camera([0.3, 0.4, 3.0], h, w, fov_deg=40.0))
    tr = _C.OptixTracer("", program, "backward.ptx")
    st = settings(bg=[0.1, 0.2, 0.3], extra=sphere_extra(samples))
    whole = gpu_forward(tr, sc, ro, rd, st)["color"]
    tr.device_status()
    rows = (1 << 16) // w  # below 131k pixels: as pairs
    if program == "envlight.ptx":  # seeded by pixel number: only the first part has the whole's
        h = rows
    for y in range(0, h, rows):
        part = gpu_forward(tr, sc, np.ascontiguousarray(ro[y:y + rows]), np.ascontiguousarray(rd[y:y + rows]), st)["color"]
        np.testing.assert_array_equal(part, whole[:, y:y + rows])
    tr.device_status()
