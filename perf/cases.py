"""Performance cases of the tracer: what its users run, through the entry
points they call, over the range of sizes and options they use.

A case is a dict of plain values. `prepare` makes what a user's program holds
before a step (scene, rays, upstream gradients, the tracer with its BVH),
`run` is one step, `work` the bytes the step cannot do without, and `exact`
the same outputs from plain torch in FP64: a pinhole rasteriser that lists
every ray's hits, sorts them by distance and composites them, differentiated
by autograd.

Kinds:
  train      one optimiser step's trace: forward and adjoint through Tracer
  render     a forward without gradients through Tracer (evaluation, viewers)
  views      refit + forward + adjoint of uneven views through ViewBatch
  secondary  forward and adjoint of the reflect / refract / environment passes
  variant    the analytic-sphere programs (forward only)
  proposal   one training step of the interval network
"""
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "diff-triangle-tracer_b200"))

DEVICE = "cuda"
# Scene families of the repository's configurations and tests: a wide cloud of
# small triangles seen from a sphere of radius 3, and a compact cloud of large
# ones under a narrow lens, where rays cross far more than one chunk of 16 hits
# and half of them end on the transmittance cut-off.
FAMILIES = {
    "cloud": {"std": 0.5, "edges": (0.005, 0.05), "fov": 50.0},
    "dense": {"std": 0.25, "edges": (0.06, 0.25), "fov": 20.0},
}
SPHERE = (0.35, 0.45, 0.0, 0.6)  # radius and centre of the variants' analytic sphere
PROPOSAL_LR, NEAR_WEIGHT, FAR_WEIGHT = 1e-3, 8.0, 3.0
REBUILD, REFIT, KEEP = 0, 1, 2


def _case(name, kind, P, H, W, **more):
    c = {"kind": kind, "P": P, "H": H, "W": W, "views": 1, "family": "cloud", "sh_degree": 3, "gas": REFIT,
         "packet": 16, "mode": "plain", "colors": "sh", "depth": 0, "samples": 0, "program": "forward"}
    if name:
        c["name"] = name
    c.update(more)
    return c


def listed():
    return [
        # a preview or a unit-sized fit: the call's own latency and its launches
        _case("preview", "render", 3000, 64, 64, gas=KEEP),
        # the small plain configuration: one 400 x 400 camera, BVH refitted each step
        _case("train_100k", "train", 100_000, 400, 400),
        # the training configuration at scale: 4 cameras stacked, tuned packets of 32 hits
        _case("train_1m_4x800", "train", 1_000_000, 800, 800, views=4, packet=32),
        # an evaluation frame of a large scene: no gradients, BVH kept
        _case("render_3m_1080p", "render", 3_000_000, 1080, 1920, gas=KEEP),
        # batched uneven views of a large scene, one graph replay a step
        _case("views_3m_x16", "views", 3_000_000, 1024, 1024, views=16, packet=32),
        # two-bounce dielectrics under an environment map
        _case("secondary_500k_2x800", "secondary", 500_000, 800, 800, views=2, depth=2),
        # odd image and scene sizes, long hit lists, degree-1 SH, and a rebuild
        # each step, as after densification changed the triangles
        _case("train_dense_rebuild", "train", 20_011, 333, 517, family="dense", sh_degree=1, gas=REBUILD),
        # exact adjoint with depth / mid-depth / distortion losses
        _case("train_exact_200k", "train", 200_000, 480, 640, mode="exact"),
        # per-triangle colours instead of SH
        _case("train_colors_300k", "train", 300_007, 512, 512, colors="rgb"),
        # cosine-sampled environment lighting off the analytic sphere
        _case("envlight_100k", "variant", 100_000, 400, 400, gas=KEEP, program="envlight", samples=8),
        # learning the proposal network: one Adam step on its standard batch
        _case("proposal_step", "proposal", 0, 1, 65_536),
        # a small secondary scene with one bounce and material gradients
        _case("secondary_20k", "secondary", 20_000, 203, 151, depth=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "render", "render", "views", "secondary", "variant", "proposal"])
    if kind == "proposal":
        return _case(None, kind, 0, 1, 128 * _log(rng, 8, 2048))  # whole tiles of 128 rays, as minibatches are
    family = "dense" if kind in ("train", "render") and rng.random() < 0.3 else "cloud"
    top = 20_000 if family == "dense" else (500_000 if kind in ("secondary", "variant") else 3_000_000)
    c = _case(None, kind, _log(rng, 1000, top), _log(rng, 24, 1080), _log(rng, 24, 1080), family=family,
              packet=rng.choice([16, 32]), sh_degree=rng.choice([0, 1, 2, 3, 3, 3]), gas=rng.choice([REBUILD, REFIT, KEEP]))
    if kind == "train":
        c["mode"] = rng.choice(["plain", "plain", "plain", "exact", "reference"])
        c["colors"] = rng.choice(["sh", "sh", "sh", "rgb"]) if c["mode"] != "reference" else "sh"
        c["views"] = rng.choice([1, 1, 2]) if family == "cloud" else 1
    elif kind == "render":
        c["mode"] = rng.choice(["plain", "plain", "reference"])
    elif kind == "views":
        c["views"] = rng.randint(2, 6)
        c["gas"] = REFIT
    elif kind == "secondary":
        c["depth"] = rng.choice([1, 2])
        c["packet"], c["gas"] = 16, REFIT
    else:
        c["program"] = rng.choice(["reflect", "refract", "envlight"])
        c["samples"] = rng.randint(1, 8) if c["program"] == "envlight" else 0
        c["packet"], c["gas"] = 16, KEEP
    return c


# ------------------------------------------------------------------ inputs
def _shapes(case):
    """Image sizes of the case's cameras; a batch's views are uneven, their
    sides 1/4, 1/2, 3/4 or all of the largest."""
    if case["kind"] != "views":
        return [(case["H"], case["W"])] * case["views"]
    part = [(1 + (5 * i + 2) % 4) for i in range(case["views"])]
    return [(max(1, case["H"] * q // 4), max(1, case["W"] * q // 4)) for q in part]


def _uniform(gen, shape, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=gen, device=DEVICE, dtype=torch.float64) * (hi - lo) + lo


def _normal(gen, shape):
    return torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float64)


def _scene(case, gen):
    """Randomly rotated triangles around normal centres; see FAMILIES."""
    P, fam = case["P"], FAMILIES[case["family"]]
    q = _normal(gen, (P, 4))
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    # the rotation's first two columns: the template triangle lies in its xy plane
    cx = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + z * w), 2 * (x * z - y * w)], 1)
    cy = torch.stack([2 * (x * y - z * w), 1 - 2 * (x * x + z * z), 2 * (y * z + x * w)], 1)
    lo, hi = fam["edges"]
    radii = torch.exp(_uniform(gen, (P, 3), math.log(lo), math.log(hi))) / math.sqrt(3.0)
    ang = torch.deg2rad(torch.tensor([90.0, 210.0, 330.0], device=DEVICE, dtype=torch.float64))
    centres = _normal(gen, (P, 3)) * fam["std"]
    verts = centres[:, None] + (radii * ang.cos())[..., None] * cx[:, None] + (radii * ang.sin())[..., None] * cy[:, None]
    M = (case["sh_degree"] + 1) ** 2
    shs = _normal(gen, (P, M, 3)) * 0.05
    shs[:, 0] = _normal(gen, (P, 3)) * 0.2 + 0.5
    return {
        "verts": verts.reshape(-1, 3).float(),
        "npts": torch.full((P,), 3, dtype=torch.int32, device=DEVICE),
        "cums": (3 * torch.arange(P, device=DEVICE)).int(),
        "opac": torch.sigmoid(_normal(gen, (P, 1))).float(),
        "sigma": _uniform(gen, (P, 1), 0.5, 2.0).float(),
        "shs": shs.float(),
        "rgb": (_normal(gen, (P, 3)) * 0.2 + 0.5).clamp(0.0, 1.0).float(),
    }


def _cameras(case, seed):
    """Pinhole cameras on a sphere of radius 3 looking at the origin:
    (origin, forward, right, up, H, W, fov in degrees), FP64."""
    rng = np.random.default_rng(seed)
    cams = []
    for H, W in _shapes(case):
        v = rng.normal(size=3)
        origin = 3.0 * v / np.linalg.norm(v)
        fwd = -origin / 3.0
        right = np.cross(fwd, [0.0, 1.0, 0.0] if abs(fwd[1]) < 0.99 else [1.0, 0.0, 0.0])
        right /= np.linalg.norm(right)
        cams.append((origin, fwd, right, np.cross(right, fwd), H, W, FAMILIES[case["family"]]["fov"]))
    return cams


def _camera_rays(cam):
    origin, fwd, right, up, H, W, fov = cam
    f64 = dict(device=DEVICE, dtype=torch.float64)
    o, fwd, right, up = (torch.tensor(a, **f64) for a in (origin, fwd, right, up))
    tan = math.tan(math.radians(fov) / 2.0)
    xs = (2.0 * (torch.arange(W, **f64) + 0.5) / W - 1.0) * tan * (W / H)
    ys = (1.0 - 2.0 * (torch.arange(H, **f64) + 0.5) / H) * tan
    d = fwd + xs[None, :, None] * right + ys[:, None, None] * up
    d = d / d.norm(dim=-1, keepdim=True)
    return o.expand(H, W, 3).float().contiguous(), d.float().contiguous()


def _upstream(case, gen, H, W):
    g = _normal(gen, (3, H, W)).float()
    go = torch.zeros((7, H, W), device=DEVICE)
    if case["mode"] == "exact":  # losses on depth, normals, mid-depth and distortion too
        go[[0, 2, 3, 4, 5, 6]] = (0.1 * _normal(gen, (6, H, W))).float()
    return g, go


def _materials(case, gen):
    P = case["P"]
    env = _uniform(gen, (1, 3, 512, 1024)).float()
    env = F.pad(F.pad(env, (0, 0, 4, 4), mode="replicate"), (4, 4, 0, 0), mode="circular")
    return {"material": (_uniform(gen, (P,)) < 0.2).int(), "ior": _uniform(gen, (P,), 1.3, 1.6).float(),
            "env": F.avg_pool2d(env, 9, 1)[0].permute(1, 2, 0).contiguous()}


def _inputs(case, seed):
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    s = {"bg": _uniform(gen, (3,)).float()}
    if case["kind"] == "proposal":
        n = case["W"]
        v = _normal(gen, (n, 3))
        o = 3.0 * v / v.norm(dim=1, keepdim=True)
        d = 0.5 * _normal(gen, (n, 3)) - o
        d = d / d.norm(dim=1, keepdim=True)
        s["rays"] = torch.cat([o, d], 1).float()
        near = 2.0 + _uniform(gen, (n, 1))
        near[_uniform(gen, (n, 1)) < 0.15] = -1.0  # rays without a hit
        s["targets"] = torch.cat([near, 3.0 + 1.5 * _uniform(gen, (n, 1))], 1).float()
        # four [rows][80] layers, He-uniform on the real inputs, zero elsewhere
        layers = []
        for rows, used, fan in ((64, 64, 78), (64, 64, 64), (64, 64, 64), (16, 2, 64)):
            w = torch.zeros((rows, 80), device=DEVICE)
            b = math.sqrt(6.0 / fan)
            w[:used, :fan] = _uniform(gen, (used, fan), -b, b).float()
            layers.append(w.reshape(-1))
        s["params"] = torch.cat(layers)
        return s
    s.update(_scene(case, gen))
    s["cams"] = _cameras(case, seed)
    if case["kind"] == "secondary":
        s.update(_materials(case, gen))
    if case["kind"] == "views":
        s["upstream"] = [_upstream(case, gen, H, W) for H, W in _shapes(case)]
    else:
        rays = [_camera_rays(c) for c in s["cams"]]  # several cameras stack into one tall image
        s["ray_o"] = torch.cat([r[0] for r in rays])
        s["ray_d"] = torch.cat([r[1] for r in rays])
        s["g"], s["go"] = _upstream(case, gen, case["views"] * case["H"], case["W"])
    return s


# ------------------------------------------------------------------ one step
def prepare(case, seed):
    import diff_tritracer
    from diff_tritracer import batch, proposal, scenes, secondary

    s = _inputs(case, seed)
    s["case"] = case
    kind, P = case["kind"], case["P"]
    if kind == "proposal":
        s["tracer"] = diff_tritracer._C.OptixTracer()
        s["net"] = proposal.Proposal(s["tracer"])
        s["net"].master.copy_(s["params"])
        s["net"].update()
        s["loss"] = torch.zeros(1, device=DEVICE)
        return s
    if kind == "views":
        tr = diff_tritracer._C.OptixTracer()
        tr.set_traversal("packets", case["packet"])
        s["cameras"] = [scenes.Camera(*c) for c in s["cams"]]
        scene = {"triangles_points": s["verts"], "sigma": s["sigma"], "num_points_per_triangle": s["npts"],
                 "cumsum_of_points_per_triangle": s["cums"], "number_of_points": P, "shs": s["shs"],
                 "opacities": s["opac"], "scaling": torch.zeros(P, device=DEVICE),
                 "density_factor": torch.zeros(P, device=DEVICE)}
        s["batch"] = batch.ViewBatch(tr, _shapes(case), scene, case["sh_degree"], s["bg"])
        return s
    if kind in ("train", "secondary"):
        for k in ("verts", "sigma", "opac", "rgb" if case["colors"] == "rgb" else "shs"):
            s[k].requires_grad_(True)
    if kind == "secondary":
        s["ior"].requires_grad_(True)
        s["env"].requires_grad_(True)
        s["tracer"] = secondary.SecondaryTracer(sh_degree=case["sh_degree"], max_depth=case["depth"])
        return s
    s["tracer"] = diff_tritracer.Tracer(case["program"] + ".ptx", "backward.ptx", exact_adjoint=case["mode"] == "exact",
                                        reference_arithmetic=case["mode"] == "reference")
    if kind != "variant":
        s["tracer"].tracer.set_traversal("packets" if case["packet"] == 32 else "auto", case["packet"])
    if case["gas"] != REBUILD:
        s["tracer"].tracer.build_tri_accel(s["verts"].detach(), s["cums"], P)
    s["settings"] = diff_tritracer.TracerSettings(
        bg=s["bg"], scale_modifier=1.0, sh_degree=case["sh_degree"], debug=False, rebuild_gas=case["gas"],
        extra_params=torch.tensor([*SPHERE, float(case["samples"])], device=DEVICE))
    s["scaling"] = torch.zeros(P, device=DEVICE)
    s["density"] = torch.zeros(P, device=DEVICE)
    return s


def _trace(s):
    rgb = s["case"]["colors"] == "rgb"
    return s["tracer"](s["ray_o"], s["ray_d"], s["verts"], s["sigma"], s["npts"], s["cums"], s["case"]["P"], s["opac"],
                       s["scaling"], s["density"], None if rgb else s["shs"], s["rgb"] if rgb else None, s["settings"])


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "proposal":
        net = s["net"]
        net.train_step(s["rays"], s["targets"], lr=PROPOSAL_LR, near_weight=NEAR_WEIGHT, far_weight=FAR_WEIGHT,
                       loss_out=s["loss"])
        return {"master": net.master, "adam_m": net.adam_m, "adam_v": net.adam_v, "loss": s["loss"]}
    if kind == "views":
        b = s["batch"]
        b.set_cameras(s["cameras"])
        b.set_upstream(s["upstream"])
        b.step()
        return {"images": [list(o) for o in b.outputs], "grads": list(b.grads), "max_blending": b.max_blending,
                "density": b.scene["density_factor"]}
    if kind == "secondary":
        color, others, maxb, scaling, density = s["tracer"](
            s["ray_o"], s["ray_d"], s["verts"], s["sigma"], s["npts"], s["cums"], case["P"], s["opac"], s["shs"],
            s["material"], s["ior"], s["env"])
        grads = torch.autograd.grad(color, [s[k] for k in ("verts", "sigma", "opac", "shs", "ior", "env")], s["g"])
        out = {"color": color, "others": others, "max_blending": maxb, "density": density, "grads": list(grads)}
    elif kind == "train":
        color, _, scaling, density, others, maxb = _trace(s)
        wrt = [s[k] for k in ("verts", "sigma", "opac", "rgb" if case["colors"] == "rgb" else "shs")]
        if case["mode"] == "exact":
            grads = torch.autograd.grad([color, others], wrt, [s["g"], s["go"]])
        else:
            grads = torch.autograd.grad(color, wrt, s["g"])
        out = {"color": color, "others": others, "max_blending": maxb, "density": density, "grads": list(grads)}
    else:
        with torch.no_grad():
            color, _, scaling, density, others, maxb = _trace(s)
        out = {"color": color, "others": others}
        if kind == "variant":  # the sphere programs write no per-triangle outputs
            return out
        out.update(max_blending=maxb, density=density)
    if case["views"] == 1:  # with several cameras, whichever blends a triangle first writes its scaling
        out["scaling"] = scaling
    return out


def work(case):
    """Bytes of one pass: rays and upstream gradients read once, images written
    once, each triangle's inputs read and its outputs written once."""
    if case["kind"] == "proposal":
        n = case["W"]
        layer = 3 * 80 * 64 + 64 * 80 * 3 + 80 * 16 * 3  # forward, input and weight gradients
        return {"bytes": 32 * n + 4 * 16640 * 6, "flops": 2 * n * layer}
    rays = sum(H * W for H, W in _shapes(case))
    per_tri = 36 + 8 + 4 * 4  # vertices, opacity and sigma, the per-triangle outputs
    coef = 12 if case["colors"] == "rgb" else 12 * (case["sh_degree"] + 1) ** 2
    per_ray = 24 + 40
    if case["kind"] in ("train", "views", "secondary"):
        per_ray += 12 + (28 if case["mode"] == "exact" else 0)
        per_tri += 36 + 8 + coef
    return {"bytes": rays * per_ray + case["P"] * (per_tri + coef), "flops": 0}


# ------------------------------------------------------------------ FP64
def exact(case, seed):
    """The outputs of `run` in FP64. None for the secondary passes (their rays
    follow no camera, so every ray would have to test every triangle) and the
    sphere programs (their bent rays are defined by FP32 expressions), and
    None for the reference-arithmetic mode, whose results are FP32 by
    definition."""
    if case["kind"] == "proposal":
        return _exact_proposal(case, seed)
    if case["kind"] in ("secondary", "variant") or case["mode"] == "reference":
        return None
    s = _inputs(case, seed)
    train = case["kind"] != "render"
    rgb = case["colors"] == "rgb"
    keys = ("verts", "sigma", "opac", "rgb" if rgb else "shs")
    leaf = {k: s[k].double().requires_grad_(train) for k in keys}
    P = case["P"]
    maxb = torch.zeros(P, device=DEVICE, dtype=torch.float64)
    images = []
    row = 0
    for i, cam in enumerate(s["cams"]):
        H, W = cam[4:6]
        if case["kind"] == "views":
            ro, rd = _camera_rays(cam)
            g, go = s["upstream"][i]
        else:
            ro, rd = s["ray_o"][row:row + H], s["ray_d"][row:row + H]
            g, go = s["g"][:, row:row + H], s["go"][:, row:row + H]
        row += H
        images.append(_exact_view(case, leaf, s["bg"].double(), cam, ro.double().reshape(-1, 3),
                                  rd.double().reshape(-1, 3), g.double().reshape(3, -1), go.double().reshape(7, -1),
                                  maxb, train))
    density = (maxb > 0).double()
    grads = [leaf[k].grad for k in keys] if train else None
    if case["kind"] == "views":
        return {"images": [list(im) for im in images], "grads": grads, "max_blending": maxb, "density": density}
    out = {"color": torch.cat([im[0] for im in images], 1), "others": torch.cat([im[1] for im in images], 1),
           "max_blending": maxb, "density": density}
    if train:
        out["grads"] = grads
    if case["views"] == 1:  # the largest angle a vertex makes with the centroid, for the triangles that blended
        rel = s["verts"].double().reshape(P, 3, 3) - s["ray_o"][0, 0].double()
        mid = rel.mean(1, keepdim=True)
        cos = (rel * mid).sum(-1) / (rel.norm(dim=-1) * mid.norm(dim=-1))
        out["scaling"] = torch.where(density > 0, cos.clamp(-1, 1).acos().amax(1), 0.0)
    return out


def _pairs(verts, cam):
    """(triangle, pixel) candidates of a pinhole camera, a block at a time:
    every pixel centre in the triangles' projected bounding boxes."""
    origin, fwd, right, up = (torch.tensor(a, device=DEVICE, dtype=torch.float64) for a in cam[:4])
    H, W, fov = cam[4:]
    tan = math.tan(math.radians(fov) / 2.0)
    rel = verts - origin
    z = rel @ fwd
    near = z < 0.05
    zs = torch.where(near, 1.0, z)
    x = ((rel @ right) / (zs * tan * W / H) + 1.0) * 0.5 * W - 0.5
    y = (1.0 - (rel @ up) / (zs * tan)) * 0.5 * H - 0.5
    some, every = near.any(1), near.all(1)

    def span(v, n):
        lo = torch.where(some, 0.0, (v.amin(1) - 1e-3).ceil().clamp(0, n))
        hi = torch.where(some, float(n - 1), (v.amax(1) + 1e-3).floor().clamp(-1, n - 1))
        return lo.long(), torch.where(every, 0.0, (hi - lo + 1).clamp(min=0)).long()

    x0, nx = span(x, W)
    y0, ny = span(y, H)
    count = nx * ny
    ends = count.cumsum(0)
    total, step, first = int(ends[-1]), 1 << 23, 0
    while first < verts.shape[0] and total:
        done = int(ends[first - 1]) if first else 0
        last = max(first + 1, int(torch.searchsorted(ends, done + step, right=True)))
        tri = torch.repeat_interleave(torch.arange(first, last, device=DEVICE), count[first:last])
        k = torch.arange(tri.numel(), device=DEVICE) - (ends[tri] - count[tri] - done)
        yield tri, (y0[tri] + k // nx[tri].clamp(min=1)) * W + x0[tri] + k % nx[tri].clamp(min=1)
        first = last


def _all_hits(verts, cam, o, d):
    """Every hit in (0, 1000]: ray, triangle and distance, sorted by ray, then distance."""
    found = []
    for tri, pix in _pairs(verts, cam):
        a, b, c = verts[tri].unbind(1)
        n = torch.linalg.cross(b - a, c - a)
        t = ((a - o[pix]) * n).sum(1) / (d[pix] * n).sum(1)
        q = o[pix] + t[:, None] * d[pix]
        inside = (t > 0) & (t <= 1000.0)
        for p0, p1 in ((a, b), (b, c), (c, a)):
            inside &= (torch.linalg.cross(p1 - p0, q - p0) * n).sum(1) >= 0
        found.append((pix[inside], tri[inside], t[inside]))
    if not found:
        empty = torch.zeros(0, dtype=torch.long, device=DEVICE)
        return empty, empty, empty.double()
    ray, tri, t = (torch.cat(x) for x in zip(*found))
    order = torch.argsort(t)
    order = order[torch.argsort(ray[order], stable=True)]
    return ray[order], tri[order], t[order]


def _sh_color(shs, degree, d):
    x, y, z = d.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    basis = [torch.full_like(x, 0.28209479177387814)]
    if degree > 0:
        basis += [-0.4886025119029199 * y, 0.4886025119029199 * z, -0.4886025119029199 * x]
    if degree > 1:
        basis += [1.0925484305920792 * x * y, -1.0925484305920792 * y * z, 0.31539156525252005 * (2 * zz - xx - yy),
                  -1.0925484305920792 * x * z, 0.5462742152960396 * (xx - yy)]
    if degree > 2:
        basis += [-0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z,
                  -0.4570457994644658 * y * (4 * zz - xx - yy), 0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy),
                  -0.4570457994644658 * x * (4 * zz - xx - yy), 1.445305721320277 * z * (xx - yy),
                  -0.5900435899266435 * x * (xx - 3 * yy)]
    return ((torch.stack(basis, 1)[..., None] * shs).sum(1) + 0.5).clamp(min=0.0)


def _shade(case, leaf, o, d, tri, train):
    """Per hit: alpha, colour, face normal and distance. The plain adjoint
    holds the hit point, the incentre distance and t constant, and passes the
    gradient through the clamp of alpha; the exact one does neither."""
    full = case["mode"] == "exact"
    a, b, c = leaf["verts"].reshape(-1, 9).index_select(0, tri).reshape(-1, 3, 3).unbind(1)
    nc = torch.linalg.cross(b - a, c - a)
    t = ((a - o) * nc).sum(1) / (d * nc).sum(1)
    q = o + t[:, None] * d
    la, lb, lc = (b - c).norm(dim=1), (c - a).norm(dim=1), (a - b).norm(dim=1)
    inc = (la[:, None] * a + lb[:, None] * b + lc[:, None] * c) / (la + lb + lc)[:, None]
    dist = None
    edge = []
    hit = q if full else q.detach()
    for p0, p1 in ((a, b), (b, c), (c, a)):
        en = F.normalize(torch.linalg.cross(nc, p0 - p1), dim=1)
        if dist is None:
            dist = (en * (inc - p0)).sum(1)
        edge.append((en * (hit - p0)).sum(1))
    phi = torch.stack(edge, 1).amax(1)
    ratio = phi / (dist if full else dist.detach())
    sigma = leaf["sigma"].reshape(-1).index_select(0, tri)
    opac = leaf["opac"].reshape(-1).index_select(0, tri)
    inside = ratio > 0
    cx = torch.where(inside, torch.where(inside, ratio, 1.0) ** sigma, 0.0)
    alpha = opac * cx
    alpha = alpha.clamp(max=0.99) if full else alpha + (alpha.clamp(max=0.99) - alpha).detach()
    if case["colors"] == "rgb":
        color = leaf["rgb"].index_select(0, tri)
    else:
        shs = leaf["shs"].reshape(leaf["shs"].shape[0], -1).index_select(0, tri).reshape(tri.numel(), -1, 3)
        color = _sh_color(shs, case["sh_degree"], F.normalize(d, dim=1))
    return alpha, color, F.normalize(nc, dim=1), t if full else t.detach()


def _exact_view(case, leaf, bg, cam, o, d, g, go, maxb, train):
    H, W = cam[4:6]
    ray, tri, t_hit = _all_hits(leaf["verts"].detach().reshape(-1, 3, 3), cam, o, d)
    counts = torch.bincount(ray, minlength=H * W)
    starts = counts.cumsum(0) - counts
    color = torch.empty((3, H * W), device=DEVICE, dtype=torch.float64)
    others = torch.zeros((7, H * W), device=DEVICE, dtype=torch.float64)
    r0 = 0
    most = 1 << 21  # hits shaded at a time
    ends = counts.cumsum(0)
    while r0 < H * W:
        base = int(starts[r0])
        r1 = max(r0 + 1, min(H * W, r0 + (1 << 18), int(torch.searchsorted(ends, base + most, right=True))))
        n = counts[r0:r1]
        hits = slice(base, base + int(n.sum()))
        with torch.set_grad_enabled(train):
            _composite(case, leaf, bg, o, d, g, go, maxb, train, color, others, r0, r1, n, starts[r0:r1] - base,
                       ray[hits], tri[hits], t_hit[hits])
        r0 = r1
    return color.reshape(3, H, W), others.reshape(7, H, W)


def _composite(case, leaf, bg, o, d, g, go, maxb, train, color, others, r0, r1, n, start, ray, tri, t_hit):
    R = r1 - r0
    # the march traces chunks of 16 hits, each starting at the last hit of the
    # one before (a closed interval): step s of a ray visits hit 15 (s / 16) + s % 16
    longest = int(n.max()) if R else 0
    s = torch.arange(max(1, 2 + longest + longest // 15), device=DEVICE)
    hit = 15 * (s // 16) + s % 16
    valid = hit[None] < n[:, None]
    flat = torch.where(valid, start[:, None] + hit[None], 0)
    if ray.numel() == 0:
        color[:, r0:r1] = bg[:, None]
        return
    alpha, rgb, normal, t = _shade(case, leaf, o[ray], d[ray], tri, train)
    valid = valid & (t_hit[flat] >= 0.2)
    a = alpha[flat]
    a = torch.where(valid & (a.detach() >= 1.0 / 255.0), a, 0.0)
    after = torch.cumsum(torch.log1p(-a), 1).exp()  # transmittance behind each step
    live = (after.detach() >= 1e-4) & (a.detach() > 0)
    a = torch.where(live, a, 0.0)
    log_t = torch.cumsum(torch.log1p(-a), 1)
    after = log_t.exp()
    w = a * torch.cat([torch.ones_like(after[:, :1]), after[:, :-1]], 1)
    last = after[:, -1]
    col = (w[..., None] * rgb[flat]).sum(1).T + last * bg[:, None]
    norm = (w[..., None] * normal[flat]).sum(1).T
    maxb.scatter_reduce_(0, tri[flat][live], w.detach()[live], "amax")
    loss = (col * g[:, r0:r1]).sum()
    color[:, r0:r1] = col.detach()
    others[1, r0:r1] = 1.0 - last.detach()
    others[2:5, r0:r1] = norm.detach()
    loss = loss + (norm * go[2:5, r0:r1]).sum()
    if case["mode"] == "exact":
        ts = t[flat]
        cw, cwt, cwtt = (torch.cumsum(v, 1) - v for v in (w, w * ts, w * ts * ts))
        depth = (w * ts).sum(1)
        distortion = (w * (ts * ts * cw - 2.0 * ts * cwt + cwtt)).sum(1)
        half = live & (after.detach() <= 0.5)
        mid = torch.where(half.any(1), ts.gather(1, half.int().argmax(1, keepdim=True))[:, 0], 0.0)
        for ch, v in ((0, depth), (5, mid), (6, distortion)):
            others[ch, r0:r1] = v.detach()
            loss = loss + (v * go[ch, r0:r1]).sum()
    if train:
        loss.backward()


def _exact_proposal(case, seed):
    """One Adam step of the interval network: 6 octaves of the closest-approach
    origin and the direction, three ReLU layers of 64, biases on a constant 1."""
    s = _inputs(case, seed)
    params = s["params"].double().requires_grad_(True)
    layers = [params[i * 64 * 80:(i + 1) * 64 * 80].reshape(-1, 80) for i in range(4)]
    rays, targets = s["rays"].double(), s["targets"].double()
    n = rays.shape[0]
    o, d = rays[:, :3], rays[:, 3:]
    off = -(o * d).sum(1, keepdim=True) / (d * d).sum(1, keepdim=True)
    v = torch.cat([(o + off * d) / 3.0, d], 1)
    enc = [v]
    for k in range(6):
        enc += [(math.pi * 2 ** k * v).sin(), (math.pi * 2 ** k * v).cos()]
    one = torch.ones((n, 1), device=DEVICE, dtype=torch.float64)
    h = torch.cat(enc + [one, 0 * one], 1)
    for w in layers[:3]:
        h = torch.cat([(h @ w.T).relu(), one, torch.zeros((n, 15), device=DEVICE, dtype=torch.float64)], 1)
    e = (h @ layers[3].T)[:, :2] - (targets - off)
    w0 = torch.where(targets[:, 0] >= 0, torch.where(e[:, 0] > 0, NEAR_WEIGHT, 1.0), 0.0)
    w1 = torch.where(e[:, 1] < 0, FAR_WEIGHT, 1.0)
    loss = (w0 * e[:, 0] ** 2 + w1 * e[:, 1] ** 2).mean()
    grad, = torch.autograd.grad(loss, params)
    m, v2 = 0.1 * grad, 0.001 * grad * grad
    master = params.detach() - PROPOSAL_LR * (m / 0.1) / ((v2 / 0.001).sqrt() + 1e-8)
    return {"master": master, "adam_m": m, "adam_v": v2, "loss": loss.detach().reshape(1)}
