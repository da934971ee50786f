"""The order of spawned secondary rays: on, off, and back to the choice by size
(which a small image over a small tree makes against sorting), told apart by
the kernels a forward launches."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import DEV, T  # noqa: E402
from scenes_for_tests import dense_scene, dense_view  # noqa: E402


def test_the_choice_by_size_can_be_restored():
    sc = dense_scene(seed=7, P=400)
    ro, rd = dense_view(H=24, W=32)
    sec = scenes.secondary_inputs(sc.P, seed=7, p_dielectric=0.3, env_shape=(32, 64), box=5)
    tr = _C.OptixTracer("", "forward.ptx", "backward.ptx")

    def launches(rebuild):
        before = tr.stats()["kernel_launches"]
        tr.trace_forward_secondary(T(ro), T(rd), T(sc.verts.reshape(-1)), T(sc.sigma), T(sc.num_points), T(sc.cumsum),
                                   sc.P, T(sc.shs), 3, T(sc.opacities), torch.zeros(sc.P, device=DEV),
                                   torch.zeros(sc.P, device=DEV), T(sec["material"]), T(sec["ior"]), T(sec["env"]), 2,
                                   rebuild)
        tr.device_status()
        return tr.stats()["kernel_launches"] - before

    launches(0)
    default = launches(2)
    tr.set_sort_secondary(True)
    assert launches(2) > default
    tr.set_sort_secondary(False)
    assert launches(2) == default
    tr.set_sort_secondary(True)
    tr.set_sort_secondary(None)
    assert launches(2) == default
