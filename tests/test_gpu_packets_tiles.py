"""Warp packets against independent lanes, bit for bit, on images of so many
tiles that no tile is taken in parts: a warp holds 32 rays, and the frustum
around them, its chords for rays of several origins, the choice between a
packet and single rays and the pairs of many rays with one triangle all run."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import DEV, T, settings  # noqa: E402

H, W = 171, 349  # 44 x 43 tiles, ragged: more than half the warps of any grid (148 SMs x 6 blocks x 4)


def _unit(v):
    return (v / np.linalg.norm(v, axis=-1, keepdims=True)).astype(np.float32)


def _pinhole(origin, fov, target=(0.0, 0.0, 0.0)):
    return scenes.camera_rays(scenes.look_at_camera(list(origin), H, W, fov_deg=fov, target=target))


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
    # origins apart, one dominant axis: packets bounded by chords wherever few triangles are there
    o = rng.uniform(-0.3, 0.3, (H, W, 3)) + [0.0, 0.0, 2.0]
    yield "scattered", (o.astype(np.float32), _unit(rng.uniform(-0.15, 0.15, (H, W, 3)) + [0.05, -0.1, -1.0]))
    (o0, d0), (o1, d1) = _pinhole([0.3, 0.4, 3.0], 6.0), _pinhole([-0.5, 0.2, 2.5], 6.0)
    odd = (np.arange(W) % 2 == 1)[None, :, None]
    yield "two_cameras", (np.where(odd, o1, o0), np.where(odd, d1, d0))
    o, d = (a.copy() for a in _pinhole([0.3, 0.4, 3.0], 6.0))
    d *= np.exp(rng.uniform(-3, 3, (H, W, 1))).astype(np.float32)  # lengths other than 1
    d[::5, ::3] = 0.0
    d[1::7, 2::4, 1] = np.nan
    d[3::9, ::5, 0] = np.inf
    o[2::6, 1::5, 0] = np.nan
    yield "broken", (o, d)


SETS = list(ray_sets())
SCENES = {
    "dense": lambda: scenes.make_scene(3000, seed=1, center_std=0.15, edge_range=(0.05, 0.3)),
    "deep": lambda: scenes.make_scene(1500, seed=2, center_std=0.05, edge_range=(0.3, 0.5)),  # buffers overflow
    "cloud": lambda: scenes.make_scene(20000, seed=5),
    "sparse": lambda: scenes.make_scene(800, seed=6, center_std=0.3, edge_range=(0.05, 0.3)),
    "one": lambda: scenes.make_scene(1, seed=7, center_std=0.01, edge_range=(0.3, 0.5)),
}


def _forward(tr, sc, ro, rd, cache, intervals=None):
    density = torch.zeros(sc.P, device=DEV)
    st = settings(bg=[0.1, 0.2, 0.3])
    buf = tr.new_hit_cache(H * W) if cache else None
    scaling = torch.zeros(sc.P, device=DEV)
    tr.build_tri_accel(T(sc.verts.reshape(-1)), T(sc.cumsum), sc.P)
    outs, maxb = tr.trace_forward_views([(T(ro), T(rd))], T(sc.verts.reshape(-1)), T(sc.sigma), T(sc.num_points),
                                        T(sc.cumsum), sc.P, T(sc.shs), 3, T(sc.opacities), scaling, density, st.bg, 2,
                                        intervals=None if intervals is None else [T(intervals)], hit_cache=buf)
    tr.device_status()
    return [x.cpu().numpy() for x in (*outs[0], density, maxb)]


def _compare(sc, ro, rd, intervals=None):
    tr = _C.OptixTracer()
    tr.set_traversal("lanes", 16, 32)
    want = _forward(tr, sc, ro, rd, False, intervals)
    for k in (16, 32):
        tr.set_traversal("packets", k)
        for cache in (False, True):  # one fused kernel; traversal pass and shading pass
            for a, b in zip(_forward(tr, sc, ro, rd, cache, intervals), want):
                np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("scene", list(SCENES))
@pytest.mark.parametrize("name,rays", SETS, ids=[s[0] for s in SETS])
def test_whole_tiles_equal_lanes(scene, name, rays):
    _compare(SCENES[scene](), *rays)


@pytest.mark.parametrize("name", ["narrow", "inside", "scattered"])
def test_clipped_tiles_equal_lanes(name):
    """Every ray its own interval: near and far ends inside the scene, none, or empty."""
    ro, rd = dict(SETS)[name]
    rng = np.random.default_rng(9)
    near = rng.uniform(0.0, 3.0, (H, W))
    iv = np.stack([np.where(rng.random((H, W)) < 0.2, -1.0, near), near + rng.uniform(-0.1, 1.0, (H, W))])
    _compare(SCENES["dense"](), ro, rd, iv.astype(np.float32))
