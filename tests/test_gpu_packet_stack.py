"""Scenes whose boxes overlap so much that a warp packet meets nearly every
node at once: its stack must hold them, or the packet be given up for its
rays one by one. A ray that loses a node would end early. Against independent
lanes, bit for bit, on images large enough that every warp takes whole
tiles of 32 rays."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import DEV, T, settings  # noqa: E402

SIDE = 256  # 2048 tiles: more than half the warps of any grid


def _pinhole(fov):
    return scenes.camera_rays(scenes.look_at_camera([0.3, 0.4, 3.0], SIDE, SIDE, fov_deg=fov))


def _unrelated():
    rng = np.random.default_rng(3)
    d = rng.normal(size=(SIDE, SIDE, 3))
    return (rng.uniform(-0.6, 0.6, (SIDE, SIDE, 3)).astype(np.float32),
            (d / np.linalg.norm(d, axis=-1, keepdims=True)).astype(np.float32))


def _deep():
    return scenes.make_scene(100_000, seed=2, center_std=0.05, edge_range=(0.3, 0.5))


def _far_triangle():
    # the Morton grid spans the far triangle too: all others share a few cells
    sc = scenes.make_scene(200_000, seed=5)
    sc.verts.reshape(-1, 3, 3)[0] += 2000.0
    return sc


CASES = {
    "deep": (_deep, lambda: _pinhole(10.0)),
    "far_triangle": (_far_triangle, lambda: _pinhole(50.0)),
    "far_triangle_unrelated_rays": (_far_triangle, _unrelated),
}


def _forward(tr, sc, ro, rd, cache):
    density = torch.zeros(sc.P, device=DEV)
    st = settings(bg=[0.1, 0.2, 0.3])
    buf = tr.new_hit_cache(SIDE * SIDE) if cache else None
    res = tr.trace_forward(T(ro), T(rd), T(sc.verts.reshape(-1)), T(sc.sigma), T(sc.num_points), T(sc.cumsum), sc.P,
                           T(sc.shs), 3, torch.empty(0, device=DEV), T(sc.opacities), torch.zeros(sc.P, device=DEV),
                           density, st.bg, st.extra_params, 0, False, hit_cache=buf)
    color, others, _, _, _, maxb = res.data
    tr.device_status()  # raises when a ray was cut short
    return [x.cpu().numpy() for x in (color, others, density, maxb)]


@pytest.mark.parametrize("case", list(CASES))
def test_no_ray_loses_nodes(case):
    scene, rays = CASES[case]
    sc = scene()
    ro, rd = rays()
    tr = _C.OptixTracer()
    tr.set_traversal("lanes", 16, 32)
    want = _forward(tr, sc, ro, rd, cache=False)
    for k in (16, 32):
        tr.set_traversal("packets", k)
        for cache in (False, True):
            for a, b in zip(_forward(tr, sc, ro, rd, cache), want):
                np.testing.assert_array_equal(a, b)
