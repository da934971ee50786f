"""The refit that follows a blob's load finds a block's tree nodes by their
number and leaf range, so tt_bvh_load has to refuse, on the host, a blob whose
ranges or numbering are not those a build gives, although its child and
parent links agree with each other."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from diff_tritracer import _C  # noqa: E402
from gpu_helpers import T  # noqa: E402
from scenes_for_tests import dense_scene  # noqa: E402
from test_gpu_bvh_blob import sections  # noqa: E402


def _views(blob):
    """Writable copies of a blob and of its tree's sections."""
    out = bytearray(blob)
    P, _, sec = sections(blob)
    view = {name: np.frombuffer(out, np.int32, sec[name][1] // 4, sec[name][0])
            for name in ("topo", "bparent", "lparent", "wsrc")}
    view["topo"] = view["topo"].reshape(-1, 4)
    return out, P, view


def _range(node, field, value):
    def edit(v, P):
        v["topo"][node, field] = value(P) if callable(value) else value
    return edit


def _both(first, last):
    def edit(v, P):
        v["topo"][0, 2:] = first, last
    return edit


def _renumber(a, b):
    """Nodes a and b swap their numbers in every link."""
    def edit(v, P):
        names = np.arange(P - 1)
        names[a], names[b] = b, a
        topo = v["topo"].copy()
        inner = topo[:, :2] >= 0
        topo[:, :2][inner] = names[topo[:, :2][inner]]
        up = v["bparent"].copy()
        up[up >= 0] = names[up[up >= 0]]
        v["topo"][names] = topo
        v["bparent"][names] = up
        v["lparent"][:] = names[v["lparent"]]
        src = v["wsrc"]
        src[src >= 0] = names[src[src >= 0]]
    return edit


def _swap_children(node):
    def edit(v, P):
        v["topo"][node, :2] = v["topo"][node, 1::-1].copy()
    return edit


def _swap_leaves(v, P):
    """Two leaves of different blocks swap places, links and all."""
    a, b = 3, P - 3
    pa, pb = int(v["lparent"][a]), int(v["lparent"][b])
    sa = 0 if v["topo"][pa, 0] == ~a else 1
    sb = 0 if v["topo"][pb, 0] == ~b else 1
    v["topo"][pa, sa], v["topo"][pb, sb] = ~b, ~a
    v["lparent"][a], v["lparent"][b] = pb, pa


EDITS = {
    "root's first leaf": _range(0, 2, 300),
    "root's range inside a block": _both(300, 400),
    "root's last leaf": _range(0, 3, lambda P: P - 2),
    "an inner node's first leaf": _range(700, 2, 10),
    "an inner node's last leaf": _range(1300, 3, lambda P: P - 1),
    "two nodes renumbered": _renumber(1, 2000),
    "neighbours renumbered": _renumber(256, 257),
    "children the wrong way round": _swap_children(0),
    "leaves out of order": _swap_leaves,
}


@pytest.fixture(scope="module")
def saved():
    sc = dense_scene(seed=2, P=2500)
    tr = _C.OptixTracer()
    tr.build_tri_accel(T(sc.verts), T(sc.cumsum), sc.P, True)
    return sc, tr.save_bvh()


@pytest.mark.parametrize("what", list(EDITS))
def test_ranges_and_numbering_are_checked(saved, what):
    sc, blob = saved
    bad, P, v = _views(blob)
    EDITS[what](v, P)
    assert bytes(bad) != bytes(blob)
    tr = _C.OptixTracer()
    with pytest.raises(RuntimeError, match="corrupted BVH blob"):
        tr.load_bvh(bytes(bad), T(sc.verts), T(sc.cumsum), sc.P)


@pytest.mark.parametrize("P", [1, 2, 3, 5, 256, 257, 2500])
def test_built_trees_load(P):
    sc = dense_scene(seed=3, P=P)
    tr = _C.OptixTracer()
    tr.build_tri_accel(T(sc.verts), T(sc.cumsum), sc.P, True)
    blob = tr.save_bvh()
    other = _C.OptixTracer()
    other.load_bvh(blob, T(sc.verts), T(sc.cumsum), sc.P)
    other.device_status()
    assert other.save_bvh() == blob
