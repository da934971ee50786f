"""Acceleration structures at the sizes where their kernels change shape: the
refit climbs 256-leaf blocks in shared memory, and a sort takes 4, 8 or 16 keys
a thread up to 32768, 65536 and more keys. A query's result depends on the
triangles alone, so the images of a refitted tree equal a fresh one's bit for
bit, and a lost or doubled triangle shows in the tree that has it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import MARGIN, gpu_forward, settings  # noqa: E402
from scenes_for_tests import dense_scene, dense_view, sphere_extra  # noqa: E402


@pytest.mark.parametrize("P", [2, 3, 255, 256, 257, 512, 513, 4095, 32768, 32769, 65536, 65537])
def test_refit_equals_build(P):
    sc = scenes.make_scene(P, seed=P, center_std=0.2, edge_range=(0.3, 0.5) if P < 16 else (0.02, 0.1))
    ro, rd = dense_view(H=45, W=67, fov=25.0)
    moved = sc.__class__(**{**sc.__dict__})
    moved.verts = (sc.verts + np.random.default_rng(P).normal(0, 0.05, sc.verts.shape)).astype(np.float32)
    tr = _C.OptixTracer("", "forward.ptx", "backward.ptx")
    first = gpu_forward(tr, sc, ro, rd, settings(rebuild=0))
    refit = gpu_forward(tr, moved, ro, rd, settings(rebuild=1))
    again = gpu_forward(tr, moved, ro, rd, settings(rebuild=1))  # the arrival flags are clear again
    tr.device_status()
    build = gpu_forward(_C.OptixTracer("", "forward.ptx", "backward.ptx"), moved, ro, rd, settings(rebuild=0))
    assert np.any(first["color"] != build["color"])
    for key in ("color", "others", "max_blending"):
        np.testing.assert_array_equal(refit[key], build[key])
        np.testing.assert_array_equal(again[key], build[key])


@pytest.mark.parametrize("h,w", [(1, 1), (3, 5), (4, 8), (5, 33)])
def test_pair_queries_at_ragged_images(oracle, h, w):
    """Bent rays are traced as (node, ray) pairs of a warp; here most warps
    have lanes without a ray. Bounds as in the full-size parity test."""
    sc = dense_scene(seed=1, P=3000)
    ro, rd = dense_view(H=h, W=w)
    bg, extra = np.array([0.1, 0.2, 0.3], np.float32), sphere_extra()
    tr = _C.OptixTracer("", "reflect.ptx", "backward.ptx")
    out = gpu_forward(tr, sc, ro, rd, settings(bg=bg, extra=extra))
    tr.device_status()
    ref = oracle.forward(sc, ro, rd, bg=bg, extra=extra, variant=1, precision=64, exact=True, canonical=True,
                         record=512, nthreads=8)
    ok = (ref.margin > MARGIN).reshape(h, w)
    want = ref.color[:, ok]
    assert np.all(np.abs(out["color"][:, ok] - want) <= 1e-5 * np.abs(want) + 1e-6)
