"""Warp packets against independent lanes, bit for bit, on rays that are no
pinhole tile: the packets cull with a frustum around their rays and take rays
one by one when it is too wide, and neither may lose or reorder a hit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import DEV, T, settings  # noqa: E402

H, W = 21, 37  # ragged against the 8x4 tile


def _unit(v):
    return (v / np.linalg.norm(v, axis=-1, keepdims=True)).astype(np.float32)


def _pinhole(origin, fov, target=(0.0, 0.0, 0.0), h=H, w=W):
    return scenes.camera_rays(scenes.look_at_camera(list(origin), h, w, fov_deg=fov, target=target))


def _parallel(direction, width):
    d = _unit(np.asarray(direction, np.float64))
    a = _unit(np.cross(d, [0.0, 1.0, 0.1]))
    b = np.cross(d, a)
    x, y = np.meshgrid(np.linspace(-width, width, W), np.linspace(-width, width, H))
    o = -3.0 * d + x[..., None] * a + y[..., None] * b
    return o.astype(np.float32), np.broadcast_to(d, o.shape).astype(np.float32).copy()


def ray_sets():
    rng = np.random.default_rng(3)
    yield "narrow", _pinhole([0.3, 0.4, 3.0], 6.0)
    yield "wide", _pinhole([0.3, 0.4, 3.0], 50.0)
    yield "axis_switch", _pinhole([2.1, 0.0, 2.1], 8.0)  # the dominant axis changes inside tiles
    yield "inside", _pinhole([0.05, 0.0, 0.02], 120.0, target=(1.0, 0.2, 0.1))
    yield "parallel", _parallel([0.2, -0.3, 1.0], 0.3)
    yield "parallel_axis", _parallel([0.0, 0.0, -1.0], 0.1)
    o = rng.uniform(-0.6, 0.6, (H, W, 3))
    yield "random", (o.astype(np.float32), _unit(rng.normal(size=(H, W, 3))))
    (o0, d0), (o1, d1) = _pinhole([0.3, 0.4, 3.0], 6.0), _pinhole([-0.5, 0.2, 2.5], 6.0)
    odd = (np.arange(W) % 2 == 1)[None, :, None]
    yield "two_cameras", (np.where(odd, o1, o0), np.where(odd, d1, d0))
    o, d = (a.copy() for a in _pinhole([0.3, 0.4, 3.0], 6.0))
    d *= np.exp(rng.uniform(-3, 3, (H, W, 1))).astype(np.float32)  # lengths other than 1
    d[::5, ::3] = 0.0
    d[1::7, 2::4, 1] = np.nan
    o[2::6, 1::5, 0] = np.nan
    yield "broken", (o, d)


SETS = list(ray_sets())
SCENES = {
    "dense": lambda: scenes.make_scene(3000, seed=1, center_std=0.15, edge_range=(0.05, 0.3)),
    "deep": lambda: scenes.make_scene(1500, seed=2, center_std=0.05, edge_range=(0.3, 0.5)),  # buffers overflow
    "cloud": lambda: scenes.make_scene(20000, seed=5),
    "one": lambda: scenes.make_scene(1, seed=7, center_std=0.01, edge_range=(0.3, 0.5)),
    "few": lambda: scenes.make_scene(33, seed=8, center_std=0.05, edge_range=(0.2, 0.5)),
}


def _forward(tr, sc, ro, rd, cache):
    P = sc.P
    density = torch.zeros(P, device=DEV)
    st = settings(bg=[0.1, 0.2, 0.3])
    buf = tr.new_hit_cache(ro.shape[0] * ro.shape[1]) if cache else None
    res = tr.trace_forward(T(ro), T(rd), T(sc.verts.reshape(-1)), T(sc.sigma), T(sc.num_points), T(sc.cumsum), P,
                           T(sc.shs), 3, torch.empty(0, device=DEV), T(sc.opacities), torch.zeros(P, device=DEV),
                           density, st.bg, st.extra_params, 0, False, hit_cache=buf)
    color, others, _, _, _, maxb = res.data
    tr.device_status()
    return [x.cpu().numpy() for x in (color, others, density, maxb)]


@pytest.mark.parametrize("scene", list(SCENES))
@pytest.mark.parametrize("name,rays", SETS, ids=[s[0] for s in SETS])
def test_packets_equal_lanes(scene, name, rays):
    sc = SCENES[scene]()
    ro, rd = rays
    tr = _C.OptixTracer()
    tr.set_traversal("lanes", 16, 32)
    want = _forward(tr, sc, ro, rd, cache=False)
    for k in (16, 32):
        tr.set_traversal("packets", k)
        for cache in (False, True):  # one fused kernel; traversal pass and shading pass
            got = _forward(tr, sc, ro, rd, cache)
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("h,w", [(1, 1), (3, 5), (4, 8), (5, 9), (1, 70)])
def test_packets_equal_lanes_at_tile_edges(h, w):
    sc = SCENES["dense"]()
    ro, rd = _pinhole([0.3, 0.4, 3.0], 5.0, h=h, w=w)
    tr = _C.OptixTracer()
    tr.set_traversal("lanes", 16, 32)
    want = _forward(tr, sc, ro, rd, cache=False)
    tr.set_traversal("packets", 16)
    for cache in (False, True):
        for a, b in zip(_forward(tr, sc, ro, rd, cache), want):
            np.testing.assert_array_equal(a, b)
