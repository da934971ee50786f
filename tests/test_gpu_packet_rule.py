"""One triangle far away makes the scene's box, and the spread of the triangles
the packet rule expects in it, as large as one likes. A packet whose frustum
then holds far more triangles than its rays meet is given up for its rays: the
work stays near that of independent lanes, and the hits are the same."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import gpu_forward, settings  # noqa: E402

SIDE = 256  # 2048 tiles: a warp holds a whole one


def _cone(common):
    rng = np.random.default_rng(3)
    o = np.zeros((SIDE, SIDE, 3)) if common else rng.uniform(-0.6, 0.6, (SIDE, SIDE, 3))
    d = rng.uniform(-0.3, 0.3, (SIDE, SIDE, 3)) + [0.0, 0.0, -1.0]
    return ((o + [0.0, 0.0, 2.0]).astype(np.float32),
            (d / np.linalg.norm(d, axis=-1, keepdims=True)).astype(np.float32))


def _counts(tr, sc, ro, rd):
    tr.reset_stats()
    out = gpu_forward(tr, sc, ro, rd, settings())
    tr.device_status()
    return out, tr.stats()


@pytest.mark.parametrize("common", [False, True], ids=["scattered", "one_origin"])
def test_wide_packets_are_given_up(common):
    sc = scenes.make_scene(100_000, seed=5)
    sc.verts.reshape(-1, 3, 3)[0] += 50.0
    ro, rd = _cone(common)
    tr = _C.OptixTracer()
    tr.set_work_counters(True)
    tr.set_traversal("lanes", 16, 32)
    want, lanes = _counts(tr, sc, ro, rd)
    for k in (16, 32):
        tr.set_traversal("packets", k)
        got, packets = _counts(tr, sc, ro, rd)
        for key in ("color", "others", "max_blending"):
            np.testing.assert_array_equal(got[key], want[key])
        # what a packet may test before it is given up, with every ray, and what its rays test then
        # (a ray of a packet of one origin tests only what its line meets)
        assert packets["triangle_tests"] < 1100 * packets["queries"] + 8 * lanes["triangle_tests"]
        # node visits: whatever a packet opens counts for each of its rays
        assert packets["node_visits"] < 4000 * packets["queries"] + 8 * lanes["node_visits"]
