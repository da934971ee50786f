"""Secondary passes sort their spawned rays by default above 2^20 pixels. On
both sides of that line the default equals both orders: images bit for bit,
gradients up to the order of float sums."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import rel_norm  # noqa: E402
from scenes_for_tests import dense_scene, dense_view  # noqa: E402
from test_gpu_secondary import gpu_secondary  # noqa: E402


@pytest.mark.parametrize("h,w", [(1024, 1024), (1024, 1025)])
def test_default_order_equals_both(h, w):
    sc = dense_scene(seed=7, P=400)
    ro, rd = dense_view(H=h, W=w, fov=40.0)
    sec = scenes.secondary_inputs(sc.P, seed=7, p_dielectric=0.3, env_shape=(32, 64), box=5)
    g, go = (np.abs(x) for x in scenes.upstream_grads(h, w, seed=13, others_std=1.0))
    outs = []
    tr = _C.OptixTracer("", "forward.ptx", "backward.ptx")
    for on in (None, True, False):  # one handle: its order buffers outlive a switch
        if on is not None:
            tr.set_sort_secondary(on)
        outs.append(gpu_secondary(tr, sc, ro, rd, sec, g, go, 1))
    for o in outs[1:]:
        for key in ("color", "others", "max_blending"):
            np.testing.assert_array_equal(o[key], outs[0][key])
        # FP32 sums of up to a million rays' terms in any order
        for x, y in zip(o["grads"], outs[0]["grads"]):
            assert rel_norm(x, y) < 1e-4
