"""What is left behind a ray's last hit is nothing: with no background its
channel sums equal the ray's outputs bit for bit, so dL/dalpha of that hit is
g T x alone, however small T is. An adjoint whose sums do not repeat the
forward's additions leaves their rounding there, a hundred times as large as
the bound here.

Every ray has its own stack of triangles, so the opacity gradient of the last
one is g x T Cx = g x w / opacity, and w is what the forward reports as the
triangle's largest blending weight."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C  # noqa: E402
from gpu_helpers import DEV, T, settings  # noqa: E402

H, W, LAYERS = 9, 13, 12
P = H * W * LAYERS
# eight FP32 roundings lie between w and the gradient, and a few in the normal
TOL = 32 * 2.0 ** -24


def _stacks():
    rng = np.random.default_rng(11)
    x, y = np.meshgrid(np.arange(W, dtype=np.float64), np.arange(H, dtype=np.float64))
    o = np.stack([x, y, np.zeros_like(x)], -1)
    d = np.zeros_like(o)
    d[..., 2] = 1.0
    # triangles of circumradius 0.35 (the rays are 1 apart), tilted, around their ray
    ang = rng.uniform(0, 2 * np.pi, (H, W, LAYERS, 1)) + np.deg2rad([0.0, 120.0, 240.0])
    tri = np.empty((H, W, LAYERS, 3, 3))
    tri[..., 0] = x[..., None, None] + 0.35 * np.cos(ang) + rng.uniform(-0.05, 0.05, (H, W, LAYERS, 1))
    tri[..., 1] = y[..., None, None] + 0.35 * np.sin(ang) + rng.uniform(-0.05, 0.05, (H, W, LAYERS, 1))
    tri[..., 2] = 2.0 + 0.4 * np.arange(LAYERS)[:, None] + rng.uniform(-0.1, 0.1, tri.shape[:-1])
    opac = rng.uniform(0.4, 0.5, (P, 1))
    cols = rng.uniform(0.2, 1.0, (P, 3))
    return (o.astype(np.float32), d.astype(np.float32), tri.reshape(P, 3, 3).astype(np.float32),
            opac.astype(np.float32), cols.astype(np.float32))


RO, RD, TRI, OPAC, COLS = _stacks()
SIGMA = np.full((P, 1), 0.3, np.float32)
LAST = np.arange(P).reshape(H, W, LAYERS)[..., -1]
C0 = 0.28209479177387814


def _shs():
    shs = np.zeros((P, 16, 3), np.float32)
    shs[:, 0] = (COLS - 0.5) / C0
    return shs


def _upstream(what):
    rng = np.random.default_rng(5)
    g, go = np.zeros((3, H, W), np.float32), np.zeros((7, H, W), np.float32)
    a, b, c = (TRI[LAST].astype(np.float64)[..., k, :] for k in range(3))
    n = np.cross(b - a, c - a)
    n /= np.linalg.norm(n, axis=-1, keepdims=True)
    if what == "color":
        g[:] = rng.uniform(0.5, 1.5, g.shape)
        col = _shs()[LAST][..., 0, :].astype(np.float64) * C0 + 0.5
        return g, go, (g.astype(np.float64) * np.moveaxis(col, -1, 0)).sum(0)
    if what == "normal":
        go[4] = rng.uniform(0.5, 1.5, (H, W))
        return g, go, go[4] * n[..., 2]
    go[0] = rng.uniform(0.5, 1.5, (H, W))
    return g, go, go[0] * ((a - RO) * n).sum(-1) / n[..., 2]  # the distance along z


def _check(maxb, dopac, gx):
    w = maxb.astype(np.float64)[LAST]
    assert (w > 1e-5).all() and (w < 1e-2).all()  # every ray blends its last layer, far behind the others
    want = gx * w / OPAC.reshape(-1).astype(np.float64)[LAST]
    got = dopac.reshape(-1).astype(np.float64)[LAST]
    assert np.abs(got / want - 1.0).max() < TOL


def _args():
    return (T(TRI.reshape(-1)), T(SIGMA), T(np.full(P, 3, np.int32)), T((3 * np.arange(P)).astype(np.int32)))


@pytest.mark.parametrize("what,mode", [("color", "plain"), ("normal", "plain"), ("color", "exact"), ("normal", "exact"),
                                       ("depth", "exact"), ("color", "reference")])
@pytest.mark.parametrize("traversal,cache", [(("packets", 16), True), (("packets", 32), True), (("packets", 16), False),
                                             (("lanes", 16), False)])
def test_last_hit_has_no_rounding_of_the_hits_before(what, mode, traversal, cache):
    tr = _C.OptixTracer(exact_adjoint=mode == "exact", reference_arithmetic=mode == "reference")
    tr.set_traversal(*traversal)
    v, sig, npts, cums = _args()
    shs, op, st = T(_shs()), T(OPAC), settings()
    buf = tr.new_hit_cache(H * W) if cache else None
    res = tr.trace_forward(T(RO), T(RD), v, sig, npts, cums, P, shs, 3, torch.empty(0, device=DEV), op,
                           torch.zeros(P, device=DEV), torch.zeros(P, device=DEV), st.bg, st.extra_params, 0, False,
                           hit_cache=buf)
    color, others, _, _, _, maxb = res.data
    g, go, gx = _upstream(what)
    bwd = tr.trace_backward(T(RO), T(RD), st.bg, v, sig, npts, cums, color, others, P, shs, 3, op, T(g), T(go),
                            torch.zeros(P, device=DEV), False, hit_cache=buf)
    tr.device_status()
    _check(maxb.cpu().numpy(), bwd.data[2].cpu().numpy(), gx)


@pytest.mark.parametrize("what", ["color", "normal"])
@pytest.mark.parametrize("exact", [False, True])
def test_last_hit_of_the_secondary_passes(what, exact):
    tr = _C.OptixTracer("", "forward.ptx", "backward.ptx", exact_adjoint=exact)
    v, sig, npts, cums = _args()
    shs, op = T(_shs()), T(OPAC)
    mat = (torch.zeros(P, dtype=torch.int32, device=DEV), torch.full((P,), 1.5, device=DEV),
           torch.zeros((8, 16, 3), device=DEV))
    color, others, maxb = tr.trace_forward_secondary(T(RO), T(RD), v, sig, npts, cums, P, shs, 3, op,
                                                     torch.zeros(P, device=DEV), torch.zeros(P, device=DEV), *mat, 1, 0)
    g, go, gx = _upstream(what)
    grads = tr.trace_backward_secondary(T(RO), T(RD), v, sig, npts, cums, color, others, P, shs, 3, op, T(g), T(go),
                                        *mat, 1)
    tr.device_status()
    _check(maxb.cpu().numpy(), grads[2].cpu().numpy(), gx)
