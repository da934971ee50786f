"""Rays whose transmittance meets the 1e-4 cut-off at the last hit of a query,
within rounding: the adjoint that replays the hit cache has to end each ray at
the hit at which the forward ended it, or it asks for a query that the forward
never made (device_status reports that)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import DEV, T, rel_norm  # noqa: E402

H, W = 96, 128


def layers(n, k):
    """n parallel triangles across the view; nearly constant opacities bring
    the transmittance behind the last visit of a ray's first query to 1e-4
    within some 1e-5 of it. (Every 16 visits the march resumes at its last hit
    and visits it again: 17 visits of 16 hits, 34 of 32.)"""
    visits = k + k // 16
    rng = np.random.default_rng(k)
    sc = scenes.make_scene(n, seed=k)
    ang = np.deg2rad(np.array([90.0, 210.0, 330.0]))[None] + rng.uniform(-0.2, 0.2, (n, 1))
    sc.verts = np.stack([2.0 * np.cos(ang), 2.0 * np.sin(ang), np.broadcast_to(-0.02 * np.arange(n)[:, None], ang.shape)],
                        axis=-1).reshape(-1, 3).astype(np.float32)
    sc.sigma = rng.uniform(1e-6, 5e-6, (n, 1)).astype(np.float32)
    sc.opacities = ((1.0 - 10.0 ** (-4.0 / visits)) / 0.4 ** sc.sigma.astype(np.float64)).astype(np.float32)
    return sc


@pytest.mark.parametrize("exact", [False, True], ids=["plain", "exact"])
@pytest.mark.parametrize("k", [16, 32])
def test_replayed_adjoint_ends_rays_as_the_forward(k, exact):
    sc = layers(k + k // 2, k)
    ro, rd = (T(x) for x in scenes.camera_rays(scenes.look_at_camera([0.0, 0.0, 3.0], H, W, fov_deg=30.0)))
    g, go = (T(np.abs(x)) for x in scenes.upstream_grads(H, W, seed=3))
    v, sig, npts, cums, shs, opac = (T(x) for x in (sc.verts.reshape(-1), sc.sigma, sc.num_points, sc.cumsum, sc.shs,
                                                    sc.opacities))
    zeros = torch.zeros(sc.P, device=DEV)
    bg = torch.zeros(3, device=DEV)
    tr = _C.OptixTracer(exact_adjoint=exact)
    tr.set_traversal("packets", k)
    tr.set_split_forward(False)  # the forward stores the queries that it makes, no others
    cache = tr.new_hit_cache(H * W, pool=2 * H * W)
    col, oth = tr.trace_forward(ro, rd, v, sig, npts, cums, sc.P, shs, 3, torch.empty(0, device=DEV), opac,
                                zeros.clone(), zeros.clone(), bg, torch.zeros(5, device=DEV), 0, False,
                                hit_cache=cache).data[:2]
    assert 0 < tr.hit_cache_usage(cache)["pool_used"] < H * W  # some rays end in their first query, others go on
    grads = []
    for c in (cache, None):
        tr.reset_stats()
        grads.append(tr.trace_backward(ro, rd, bg, v, sig, npts, cums, col, oth, sc.P, shs, 3, opac, g, go,
                                       zeros.clone(), False, hit_cache=c).data)
        tr.device_status()
    # FP32 sums of up to 12288 rays' terms in any order, ~1e-6, and S in another order than ray by ray
    for a, b in zip(*grads):
        assert rel_norm(a.cpu().numpy(), b.cpu().numpy()) < 1e-4
