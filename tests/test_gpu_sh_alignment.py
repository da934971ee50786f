"""SH coefficients and their gradients may lie at any float of a larger buffer
(a view of one flat parameter or gradient vector): the kernels take them 16
bytes at a time only where both start on such a boundary."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():  # collected on CPU hosts, skipped there
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C, scenes  # noqa: E402
from gpu_helpers import DEV, T, rel_norm, settings  # noqa: E402
from scenes_for_tests import dense_scene, dense_view, sphere_extra  # noqa: E402

H, W = 48, 64
SC = dense_scene(seed=4, P=1500)
RAYS = dense_view(H, W)


def _at(shape, offset, fill=None):
    """A [*shape] view that starts `offset` floats into its buffer."""
    n = int(np.prod(shape))
    flat = torch.zeros(n + 8, device=DEV)
    view = flat[offset:offset + n].view(shape)
    if fill is not None:
        view.copy_(fill)
    assert view.data_ptr() % 16 == 4 * (offset % 4)
    return view


def _scene(shs):
    return (T(SC.verts.reshape(-1)), T(SC.sigma), T(SC.num_points), T(SC.cumsum), SC.P, shs, 3, T(SC.opacities),
            torch.zeros(SC.P, device=DEV), torch.zeros(SC.P, device=DEV))


def _plain(sh_off, grad_off, cache, traversal):
    tr = _C.OptixTracer()
    tr.set_traversal(*traversal)
    v, sig, npts, cums, P, shs, deg, op, scal, dens = _scene(_at((SC.P, 16, 3), sh_off, T(SC.shs)))
    st = settings(bg=[0.1, 0.2, 0.3])
    ro, rd = T(RAYS[0]), T(RAYS[1])
    buf = tr.new_hit_cache(H * W) if cache else None
    res = tr.trace_forward(ro, rd, v, sig, npts, cums, P, shs, deg, torch.empty(0, device=DEV), op, scal, dens, st.bg,
                           st.extra_params, 0, False, hit_cache=buf)
    color, others = res.data[:2]
    g, go = (T(x) for x in scenes.upstream_grads(H, W, seed=1, others_std=1.0))
    grads = (torch.empty_like(v), torch.empty_like(sig), torch.empty_like(op), _at((P, 16, 3), grad_off))
    tr.trace_backward_views([(ro, rd)], [(color, others)], [(g, go)], v, sig, npts, cums, P, shs, deg, op, st.bg,
                            grads=grads, hit_cache=buf)
    tr.device_status()
    return [x.cpu().numpy() for x in (color, others, *grads)]


# float sums of a few thousand terms in any order: 2^-24 times the root of
# their number, with room for cancellation among them
TOL = 1e-4


@pytest.mark.parametrize("cache", [True, False])
@pytest.mark.parametrize("traversal", [("packets", 16), ("packets", 32), ("lanes", 16)])
def test_plain_passes_take_any_alignment(traversal, cache):
    want = _plain(0, 0, cache, traversal)
    for offs in ((1, 0), (0, 3), (2, 1), (4, 4)):
        got = _plain(*offs, cache, traversal)
        for a, b in zip(got[:2], want[:2]):
            np.testing.assert_array_equal(a, b)
        for a, b in zip(got[2:], want[2:]):
            assert rel_norm(a, b) < TOL


def test_secondary_passes_take_any_alignment():
    sec = scenes.secondary_inputs(SC.P, seed=7, p_dielectric=0.3, env_shape=(32, 64), box=5)
    g, go = (T(x) for x in scenes.upstream_grads(H, W, seed=1, others_std=1.0))

    def run(off):
        tr = _C.OptixTracer("", "forward.ptx", "backward.ptx")
        v, sig, npts, cums, P, shs, deg, op, scal, dens = _scene(_at((SC.P, 16, 3), off, T(SC.shs)))
        ro, rd = T(RAYS[0]), T(RAYS[1])
        mat = [T(sec[k]) for k in ("material", "ior", "env")]
        color, others, _ = tr.trace_forward_secondary(ro, rd, v, sig, npts, cums, P, shs, deg, op, scal, dens, *mat, 2, 0)
        grads = tr.trace_backward_secondary(ro, rd, v, sig, npts, cums, color, others, P, shs, deg, op, g, go, *mat, 2,
                                            material_grads=True)
        tr.device_status()
        return [x.cpu().numpy() for x in (color, others, *grads)]

    want = run(0)
    for off in (1, 2):
        got = run(off)
        for a, b in zip(got[:2], want[:2]):
            np.testing.assert_array_equal(a, b)
        for a, b in zip(got[2:], want[2:]):
            assert rel_norm(a, b) < TOL


@pytest.mark.parametrize("program", ["reflect.ptx", "envlight.ptx"])
def test_sphere_programs_take_any_alignment(program):
    def run(off):
        tr = _C.OptixTracer("", program, "backward.ptx")
        v, sig, npts, cums, P, shs, deg, op, scal, dens = _scene(_at((SC.P, 16, 3), off, T(SC.shs)))
        st = settings(bg=[0.1, 0.2, 0.3], extra=sphere_extra())
        res = tr.trace_forward(T(RAYS[0]), T(RAYS[1]), v, sig, npts, cums, P, shs, deg, torch.empty(0, device=DEV), op,
                               scal, dens, st.bg, st.extra_params, 0, False)
        tr.device_status()
        return res.data[0].cpu().numpy()

    np.testing.assert_array_equal(run(1), run(0))
