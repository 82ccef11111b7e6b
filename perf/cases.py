"""Performance cases of the render-and-train path: what each is, its inputs, one pass of it
through the public entry points of splatrs_b200.gpu, the work it cannot do without, and its
result in 64 bits by plain torch.

Kinds
  view    project_all -> bin -> rasterize_forward of one view (a viewer's frame, an
          evaluation render).
  step    the same plus rasterize_backward and project_backward_all: parameter gradients of
          one view, as a custom training loop takes them.
  host    Renderer.render_backward: the same chain driven with host buffers.
  loss    photometric_loss of an image against an 8-bit or float target, with its gradient.
  train   Trainer.run and the updated model: one view per iteration, or `batch` views.
  policy  the learned-densification network: probabilities of every Gaussian and one
          training gradient on a subset of records.
Scenes are synthetic, with the shapes and distributions of splatrs_b200/scenes.py.
"""
import ctypes
import math

import numpy as np
import torch

from splatrs_b200 import gpu as G
from splatrs_b200._lib import Camera, ProjOpts
from splatrs_b200.scenes import look_at

_ctx = None


def _context():
    """The program's one context for the stage entry points."""
    global _ctx
    if _ctx is None:
        _ctx = G.Context(0)
    return _ctx


def listed():
    return [
        # A 256x256 thumbnail of a 10k-Gaussian scene: latency and launches.
        dict(name="view-256", kind="view", scene="blobs", n=10000, width=256, height=256, sh=3, antialias=False),
        # An evaluation or viewer frame of a large scene at full HD.
        dict(name="view-1080p", kind="view", scene="box", n=1000000, width=1920, height=1080, sh=3, antialias=False),
        # The smallest differentiable step: gradient checks, toy fits.
        dict(name="step-128x96", kind="step", scene="blobs", n=2000, width=128, height=96, sh=3, antialias=False),
        # A sparse scene at 720p with the anti-aliased opacity compensation.
        dict(name="step-720p", kind="step", scene="box", n=100000, width=1280, height=720, sh=3, antialias=True),
        # A trained clustered scene at the dataset's odd size, before the last SH degree.
        dict(name="step-1297x840", kind="step", scene="shells", n=187001, width=1297, height=840, sh=2,
             antialias=False),
        # The render benchmark: one million Gaussians, full HD, forward and backward.
        dict(name="step-1080p", kind="step", scene="box", n=1000000, width=1920, height=1080, sh=3, antialias=False),
        # A host program that holds its images and gradients in host memory.
        dict(name="host-1297x840", kind="host", scene="shells", n=100000, width=1297, height=840, sh=3,
             antialias=False),
        # The loss of a training view by itself (an evaluation, another renderer's image).
        dict(name="loss-1297x840", kind="loss", width=1297, height=840, u8=True),
        # Training the small multi-view scene once it has grown: 256x256 views.
        dict(name="train-blobs", kind="train", scene="blobs", n=34380, width=256, height=256, views=16, batch=1,
             iterations=30, bf16=False, fp64_conic=False),
        # Training the clustered scene at 1297x840 at its converged size.
        dict(name="train-shells", kind="train", scene="shells", n=187001, width=1297, height=840, views=6, batch=1,
             iterations=20, bf16=False, fp64_conic=False),
        # Batched mixed-size training: 8 views a step, BF16 storage, f64 conics.
        dict(name="train-batch", kind="train", scene="shells", n=100000, width=0, height=0, views=12, batch=8,
             iterations=4, bf16=True, fp64_conic=True),
        # Learned densification at an event: all Gaussians scored, one gradient of 65,536 records.
        dict(name="policy-500k", kind="policy", n=500000, records=65536),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("view", "view", "step", "step", "step", "host", "loss", "train", "train", "policy"))
    if kind == "policy":
        n = _log_int(rng, 1000, 1000000)
        return dict(kind=kind, n=n, records=min(n, _log_int(rng, 1000, 65536)))
    width = _log_int(rng, 64, 1920)
    height = max(48, min(1080, int(width * rng.uniform(0.5, 1.0))))
    if kind == "loss":
        return dict(kind=kind, width=width, height=height, u8=rng.random() < 0.75)
    scene = rng.choice(("blobs", "box", "shells"))
    if kind == "train":
        width, height = max(128, width * 2 // 3), max(96, height * 2 // 3)
        if rng.random() < 0.3:
            return dict(kind=kind, scene=scene, n=_log_int(rng, 2000, 100000 if scene != "blobs" else 35000), width=0,
                        height=0, views=9, batch=rng.randint(2, 8), iterations=4, bf16=True, fp64_conic=True)
        return dict(kind=kind, scene=scene, n=_log_int(rng, 2000, 187000 if scene != "blobs" else 35000), width=width,
                    height=height, views=rng.randint(3, 12), batch=1, iterations=rng.randint(10, 20),
                    bf16=rng.random() < 0.25, fp64_conic=rng.random() < 0.25)
    most = {"blobs": 35000, "box": 1000000, "shells": 500000}[scene]
    if kind == "host":
        most = min(most, 200000)
    return dict(kind=kind, scene=scene, n=_log_int(rng, 1000, most), width=width, height=height,
                sh=rng.choice((0, 1, 2, 3, 3, 3)), antialias=rng.random() < 0.25)


# ---------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)


def _normal(gen, mu, sigma, *shape):
    return torch.empty(shape, device="cuda").normal_(mu, sigma, generator=gen)


def _uniform(gen, lo, hi, *shape):
    return torch.empty(shape, device="cuda").uniform_(lo, hi, generator=gen)


def _log_scale(scene, n):
    """(mean, standard deviation) of the log-scales: the shells' Gaussians cover their
    surfaces, so fewer are larger."""
    if scene == "blobs":
        return -4.0, 0.3
    if scene == "box":
        return -4.5, 0.5
    return -4.5 + 0.5 * math.log(500000 / max(n, 20000)), 0.3


def _gaussians(scene, n, gen):
    """(n, 59) reference records on the GPU."""
    g = torch.empty((n, 59), device="cuda")
    if scene == "blobs":
        g[:, 0:3] = _uniform(gen, -1.0, 1.0, n, 3)
    elif scene == "box":
        g[:, 0:3] = _uniform(gen, -5.0, 5.0, n, 3)
    else:
        shells = 40
        radius = _uniform(gen, 0.2, 2.0, shells)
        planar = _uniform(gen, 0.0, 1.0, shells) < 0.5
        centre = _uniform(gen, -1.0, 1.0, shells, 3) * (3.0 - radius)[:, None]
        normal = _normal(gen, 0.0, 1.0, shells, 3)
        normal /= normal.norm(dim=1, keepdim=True)
        area = torch.where(planar, 1.0, 4.0) * radius ** 2
        edges = torch.cumsum(area / area.sum(), 0)
        s = torch.searchsorted(edges, _uniform(gen, 0.0, 1.0, n)).clamp_(max=shells - 1)
        d = _normal(gen, 0.0, 1.0, n, 3)
        flat = d - (d * normal[s]).sum(1, keepdim=True) * normal[s]
        flat = flat / flat.norm(dim=1, keepdim=True) * _uniform(gen, 0.0, 1.0, n, 1).sqrt()
        d = torch.where(planar[s][:, None], flat, d / d.norm(dim=1, keepdim=True))
        g[:, 0:3] = centre[s] + radius[s][:, None] * d + _normal(gen, 0.0, 0.01, n, 3)
    mu, sigma = _log_scale(scene, n)
    g[:, 3:6] = _normal(gen, mu, sigma, n, 3)
    q = _normal(gen, 0.0, 1.0, n, 4)
    g[:, 6:10] = q / q.norm(dim=1, keepdim=True)
    g[:, 10] = _normal(gen, 0.0, 1.5 if scene == "box" else 1.0, n)
    g[:, 11:14] = _normal(gen, 0.5, 0.2, n, 3)
    g[:, 14:59] = _normal(gen, 0.0, 0.05, n, 45)
    return g


def _focal(scene, width, height):
    if scene == "blobs":
        return 300.0 / 256.0 * min(width, height)
    if scene == "box":
        return 1500.0 / 1920.0 * width
    return 1150.0 / 1297.0 * width


def _distance(scene):
    return {"blobs": 4.0, "box": 12.0, "shells": 8.0}[scene]


def _camera(scene, width, height, angle, lift=-0.3):
    """A camera at `angle` (radians) around the vertical axis, `lift` below zero is above."""
    r = _distance(scene)
    h = lift * r
    ring = math.sqrt(r * r - h * h)
    f = _focal(scene, width, height)
    return Camera.from_record(look_at(width, height, f, f, (ring * math.sin(angle), h, -ring * math.cos(angle)),
                                      (0.0, 0.0, 0.0)))


def _angle(seed):
    return 0.7 * (int(seed) % 9)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if kind == "loss":
        npix = case["width"] * case["height"]
        target = _uniform(gen, 0.0, 1.0, npix * 3)
        pred = target + _normal(gen, 0.0, 0.05, npix * 3)
        if case["u8"]:
            target = (target * 255.0).round().to(torch.uint8)
        return dict(case=case, pred=pred, target=target)
    if kind == "policy":
        n, m = case["n"], case["records"]
        theta = torch.zeros(16 * 64 + 64 + 64 * 64 + 64 + 64 * 3 + 3, device="cuda")
        o = 0
        for a, b in ((16, 64), (64, 64), (64, 3)):
            lim = math.sqrt(6.0 / (a + b))
            theta[o:o + a * b] = _uniform(gen, -lim, lim, a * b)
            o += a * b + b
        return dict(case=case, x=_normal(gen, 0.0, 1.0, n, 16), theta=theta,
                    rx=_normal(gen, 0.0, 1.0, m, 16),
                    ry=torch.randint(0, 3, (m,), device="cuda", generator=gen, dtype=torch.int32),
                    rw=_uniform(gen, 0.2, 2.0, m))
    g = _gaussians(case["scene"], case["n"], gen)
    if kind == "train":
        return _prepare_train(case, seed, gen, g)
    w, h = case["width"], case["height"]
    cam = _camera(case["scene"], w, h, _angle(seed))
    opts = ProjOpts.make(sh_degree=case["sh"], antialias=case["antialias"])
    state = dict(case=case, n=case["n"], cam=cam, opts=opts, bg=(0.1, 0.2, 0.3))
    if kind != "view":
        state["dimage"] = _normal(gen, 0.0, 1.0, w * h * 3)
    if kind == "host":
        ctx = G.Context(0)
        rend = G.Renderer(ctx)
        rend.set_model(g.cpu().numpy(), case["sh"])
        pinned = lambda *shape: torch.empty(shape, pin_memory=True)  # noqa: E731
        d = pinned(w * h * 3)
        d.copy_(state.pop("dimage"))
        state.update(ctx=ctx, rend=rend, dimage=d.numpy(), image=pinned(w * h * 3).numpy(),
                     grads=pinned(case["n"], 59).numpy(), keep=d)
    else:
        state.update(ctx=_context(), planes=G.params_to_planes(_context(), g))
    return state


_MIXED = ((640, 480), (1024, 768), (1297, 840), (1600, 1200))


def _prepare_train(case, seed, gen, truth):
    """A trainer near the end of its schedule: views rendered from `truth`, the model a
    perturbed `truth`, all rates a hundredth of the defaults (as the position rate has
    decayed by then), no densification."""
    n, scene = case["n"], case["scene"]
    ctx = _context()
    planes = G.params_to_planes(ctx, truth)
    views = []
    for k in range(case["views"]):
        w, h = (case["width"], case["height"]) if case["width"] else _MIXED[k % 4]
        cam = _camera(scene, w, h, _angle(seed) + 2.399963 * k, -0.1 - 0.6 * k / case["views"])
        proj = G.project_all(ctx, planes, n, n, cam, ProjOpts.make(sh_degree=3))
        out = G.rasterize_forward(ctx, proj, G.bin(ctx, proj), (0.0, 0.0, 0.0), count_pairs=False)
        views.append((cam, (out.image.clamp(0.0, 1.0) * 255.0).round().to(torch.uint8).cpu().numpy()))
    model = truth.clone()
    model[:, 0:3] += _normal(gen, 0.0, 0.003, n, 3)
    model[:, 3:6] += _normal(gen, 0.0, 0.05, n, 3)
    model[:, 10] += _normal(gen, 0.0, 0.1, n)
    model[:, 11:14] += _normal(gen, 0.0, 0.03, n, 3)
    own = G.Context(0)
    trainer = G.Trainer(own, model.cpu().numpy(), 1.1 * _distance(scene), views, densify=0, sh_degree_interval=1,
                        seed=int(seed), batch_views=case["batch"], bf16_storage=int(case["bf16"]),
                        fp64_conic=int(case["fp64_conic"]), position_lr_init=1.6e-6, position_lr_final=1.6e-6,
                        feature_lr=2.5e-5, opacity_lr=1e-4, scaling_lr=5e-5, rotation_lr=1e-5)
    trainer.run(6)  # past the SH schedule
    return dict(case=case, ctx=own, trainer=trainer)


# ---------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "loss":
        out, grad = G.photometric_loss(_context(), state["pred"], state["target"], case["width"], case["height"], 0.2)
        return out, grad
    if kind == "policy":
        ctx = _context()
        prob = G.mlp_forward(ctx, state["x"], state["theta"], tcgen05=True)
        grad = G.mlp_grad(ctx, state["rx"], state["ry"], state["rw"], state["theta"], tcgen05=True)
        return prob, grad
    if kind == "train":
        info = state["trainer"].run(case["iterations"])
        return info["loss"], state["trainer"].model()
    if kind == "host":
        return state["rend"].render_backward(state["cam"], state["opts"], state["bg"], state["dimage"],
                                             state["image"], state["grads"])
    ctx, n = state["ctx"], state["n"]
    proj = G.project_all(ctx, state["planes"], n, n, state["cam"], state["opts"])
    b = G.bin(ctx, proj)
    out = G.rasterize_forward(ctx, proj, b, state["bg"], count_pairs=False)
    if kind == "view":
        return out.image, out.final_t, out.n_contrib
    pgrad = G.rasterize_backward(ctx, proj, b, state["bg"], out, state["dimage"])
    grads = G.project_backward_all(ctx, state["planes"], n, n, state["cam"], state["opts"], proj, pgrad)
    return out.image, out.final_t, out.n_contrib, pgrad, grads


# ---------------------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------------------
def _pairs(scene, n, width, height):
    """Expected (Gaussian, pixel) pairs above the alpha threshold: every Gaussian's ellipse
    2 pi sigma_max times the mean of its squared pixel size, sigma_max = ln(255 opacity)."""
    mu, sigma = _log_scale(scene, n)
    f = _focal(scene, width, height) / _distance(scene)
    var = f * f * math.exp(2.0 * mu + 2.0 * sigma * sigma) + 0.3
    return n * min(2.0 * math.pi * 4.7 * var, float(width) * height)


def work(case):
    kind = case["kind"]
    if kind == "loss":
        px = case["width"] * case["height"]
        return {"bytes": px * (12 + (3 if case["u8"] else 12) + 12), "flops": px * 1056}
    if kind == "policy":
        return {"bytes": case["n"] * 76 + case["records"] * 72,
                "flops": case["n"] * 10624 + case["records"] * 31872}
    if kind == "train":
        if case["width"]:
            sizes = [(case["width"], case["height"])] * case["batch"]
        else:
            sizes = [_MIXED[k % 4] for k in range(case["batch"])]
        px = sum(w * h for w, h in sizes)
        pairs = sum(_pairs(case["scene"], case["n"], w, h) for w, h in sizes)
        n = case["n"]
        return {"bytes": case["iterations"] * (n * (3 * 2 * 236) + px * 3) + n * 236,
                "flops": case["iterations"] * (pairs * 70 + px * 1056)}
    px = case["width"] * case["height"]
    pairs = _pairs(case["scene"], case["n"], case["width"], case["height"])
    read = (11 + 3 * (case["sh"] + 1) ** 2) * 4
    if kind == "view":
        return {"bytes": case["n"] * read + px * 20, "flops": pairs * 20}
    if kind == "host":
        return {"bytes": case["n"] * (read + 236) + px * 24, "flops": pairs * 70}
    return {"bytes": case["n"] * (read + 240 + 48) + px * 32, "flops": pairs * 70}


# ---------------------------------------------------------------------------------------
# The results in 64 bits
# ---------------------------------------------------------------------------------------
_C1 = 0.4886025119029199
_C2 = (1.0925484305920792, -1.0925484305920792, 0.31539156525252005, -1.0925484305920792, 0.5462742152960396)
_C3 = (-0.5900435899266435, 2.890611442640554, -0.4570457994644658, 0.3731763325901154, -0.4570457994644658,
       1.445305721320277, -0.5900435899266435)


def _basis64(d, degree):
    x, y, z = d.unbind(1)
    b = [torch.full_like(x, 0.28209479177387814)]
    if degree >= 1:
        b += [-_C1 * y, _C1 * z, -_C1 * x]
    if degree >= 2:
        b += [_C2[0] * x * y, _C2[1] * y * z, _C2[2] * (2 * z * z - x * x - y * y), _C2[3] * x * z,
              _C2[4] * (x * x - y * y)]
    if degree >= 3:
        b += [_C3[0] * y * (3 * x * x - y * y), _C3[1] * x * y * z, _C3[2] * y * (4 * z * z - x * x - y * y),
              _C3[3] * z * (2 * z * z - 3 * x * x - 3 * y * y), _C3[4] * x * (4 * z * z - x * x - y * y),
              _C3[5] * z * (x * x - y * y), _C3[6] * x * (x * x - 3 * y * y)]
    return torch.stack(b, 1)


def _project64(p, cam, opts):
    """Projection of (n, 59) float64 records: indices of the visible Gaussians and, for those,
    mean2d, conic, opacity, colour, depth and the 16-pixel tile rectangle."""
    dev = p.device
    as64 = lambda v: torch.tensor(v, dtype=torch.float64, device=dev)  # noqa: E731
    R, tr = as64(list(cam.rot)).reshape(3, 3), as64(list(cam.trans))
    fx, fy, cx, cy, W, H = cam.fx, cam.fy, cam.cx, cam.cy, cam.width, cam.height
    near = opts.near_plane
    front = torch.nonzero((p[:, 0:3].detach() @ R.T + tr)[:, 2] > near).squeeze(1)
    g = p[front]
    t = g[:, 0:3] @ R.T + tr
    s = g[:, 3:6].exp()
    q = g[:, 6:10]
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                       2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                       2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    m = rot * s[:, None, :]
    rz = 1 / t[:, 2]
    rx, ry = t[:, 0] * rz, t[:, 1] * rz
    tan_x, tan_y = 0.5 * W / fx, 0.5 * H / fy
    rxc = rx.clamp(-(cx / fx + 0.3 * tan_x), (W - cx) / fx + 0.3 * tan_x)
    ryc = ry.clamp(-(cy / fy + 0.3 * tan_y), (H - cy) / fy + 0.3 * tan_y)
    zero = torch.zeros_like(rz)
    jac = torch.stack([fx * rz, zero, -fx * rxc * rz, zero, fy * rz, -fy * ryc * rz], 1).reshape(-1, 2, 3)
    tm = (jac @ R) @ m
    cov = tm @ tm.transpose(1, 2)
    a0, b, c0 = cov[:, 0, 0], cov[:, 0, 1], cov[:, 1, 1]
    a, c = a0 + opts.eps2d, c0 + opts.eps2d
    det = a * c - b * b
    conic = torch.stack([c / det, -b / det, a / det], 1)
    opacity = torch.sigmoid(g[:, 10])
    if opts.antialias:
        opacity = opacity * ((a0 * c0 - b * b).clamp(min=1e-300) / det).sqrt()
    mean2d = torch.stack([fx * rx + cx, fy * ry + cy], 1)
    d = g[:, 0:3] + R.T @ tr
    d = d / d.norm(dim=1, keepdim=True)
    k = (opts.sh_degree + 1) ** 2
    sh = g[:, 11:59].reshape(-1, 16, 3)
    color = (0.5 + (_basis64(d, opts.sh_degree)[:, :, None] * sh[:, :k]).sum(1)).clamp(min=0)
    with torch.no_grad():
        mid = 0.5 * (a + c)
        radius = (3 * (mid + (mid * mid - det).clamp(min=0.1).sqrt()).sqrt()).ceil()
        tx, ty = (W + 15) // 16, (H + 15) // 16
        lo = ((mean2d - radius[:, None]) / 16).floor().clamp(min=0)
        hi = ((mean2d + radius[:, None]) / 16).ceil()
        hi = torch.stack([hi[:, 0].clamp(0, tx), hi[:, 1].clamp(0, ty)], 1)
        seen = torch.nonzero((det > 0) & (lo < hi).all(1)).squeeze(1)
        tiles = torch.cat([lo, hi], 1)[seen].long()
    return front[seen], mean2d[seen], conic[seen], opacity[seen], color[seen], t[seen, 2], tiles


def _composite64(mean2d, conic, opacity, color, depth, tiles, width, height, bg, most):
    """Front-to-back compositing of all (Gaussian, pixel) pairs: image, final transmittance,
    and per pair (Gaussian, sigma, A dx + B dy, B dx + C dy, weight); None over `most` pairs."""
    dev = mean2d.device
    with torch.no_grad():
        order = torch.argsort(depth, stable=True)
        smax = (255 * opacity).log()
        det = conic[:, 0] * conic[:, 2] - conic[:, 1] ** 2
        half = (2 * smax.clamp(min=0)[:, None] * torch.stack([conic[:, 2], conic[:, 0]], 1) / det[:, None]).sqrt() + 1e-3
        size = torch.tensor([width, height], dtype=torch.float64, device=dev)
        lo = torch.maximum((mean2d - half - 0.5).ceil().clamp(min=0), tiles[:, 0:2] * 16.0)
        hi = torch.minimum(torch.minimum((mean2d + half - 0.5).floor() + 1, size), tiles[:, 2:4] * 16.0)
        ext = (hi - lo).clamp(min=0).long() * (smax > 0)[:, None]
        lo = lo.long()
        cnt = (ext[:, 0] * ext[:, 1])[order]
        total = int(cnt.sum())
        if total > most:
            return None
        g = order.repeat_interleave(cnt)
        k = torch.arange(total, device=dev) - (cnt.cumsum(0) - cnt).repeat_interleave(cnt)
        px, py = lo[g, 0] + k % ext[g, 0], lo[g, 1] + k // ext[g, 0]
        dx, dy = px + 0.5 - mean2d[g, 0], py + 0.5 - mean2d[g, 1]
        sig = 0.5 * (conic[g, 0] * dx * dx + conic[g, 2] * dy * dy) + conic[g, 1] * dx * dy
        keep = (sig >= 0) & (sig <= smax[g]) & (opacity[g] * (-sig).exp() >= 1 / 255)
        g, pix = g[keep], (py * width + px)[keep]
        del k, px, py, dx, dy, sig, keep
        pix, perm = torch.sort(pix, stable=True)
        g = g[perm]
        del perm
        px, py = (pix % width).double() + 0.5, (pix // width).double() + 0.5
    dx, dy = px - mean2d[g, 0], py - mean2d[g, 1]
    gx, gy = conic[g, 0] * dx + conic[g, 1] * dy, conic[g, 1] * dx + conic[g, 2] * dy
    sigma = 0.5 * (gx * dx + gy * dy)
    alpha = (opacity[g] * (-sigma).exp()).clamp(max=0.99)
    la = torch.log1p(-alpha)
    after = la.cumsum(0)
    first = torch.searchsorted(pix, pix)  # each pair's first pair of its pixel
    before = (after - la) - (after - la)[first]
    live = (before + la).detach().exp() >= 1e-4
    weight = torch.where(live, alpha * before.exp(), 0.0)
    npix = width * height
    image = torch.zeros((npix, 3), dtype=torch.float64, device=dev).index_add(0, pix, weight[:, None] * color[g])
    ft = torch.zeros(npix, dtype=torch.float64, device=dev).index_add(0, pix, torch.where(live, la, 0.0)).exp()
    image = image + ft[:, None] * torch.tensor(bg, dtype=torch.float64, device=dev)
    return image.reshape(-1), ft, (g, sigma, gx.detach(), gy.detach(), weight.detach())


def _planes64(aos):
    """Parameter planes (15, n, 4) of (n, 59) records."""
    n = aos.shape[0]
    z = torch.zeros((n, 1), dtype=aos.dtype, device=aos.device)
    p = torch.cat([aos[:, 0:3], aos[:, 10:11], aos[:, 6:10], aos[:, 3:6], z, aos[:, 11:59]], 1)
    return p.reshape(n, 15, 4).permute(1, 0, 2).reshape(-1)


def _f32(v):
    """The value that the entry points receive: options and cameras hold f32."""
    return ctypes.c_float(v).value


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return None
    if kind == "loss":
        return _exact_loss(case, prepare(case, seed))
    if kind == "policy":
        return _exact_policy(prepare(case, seed))
    gen = _generator(seed)
    w, h, n = case["width"], case["height"], case["n"]
    aos = _gaussians(case["scene"], n, gen).double()
    dimage = _normal(gen, 0.0, 1.0, w * h * 3).double() if kind != "view" else None
    cam = _camera(case["scene"], w, h, _angle(seed))
    opts = ProjOpts.make(sh_degree=case["sh"], antialias=case["antialias"])
    bg = tuple(_f32(v) for v in (0.1, 0.2, 0.3))
    aos.requires_grad_(kind != "view")
    idx, mean2d, conic, opacity, color, depth, tiles = _project64(aos, cam, opts)
    screen = [v.detach().requires_grad_(kind != "view") for v in (mean2d, conic, opacity, color)]
    got = _composite64(*screen, depth.detach(), tiles, w, h, bg, 150_000_000)
    if got is None:
        return None
    image, ft, (g, sigma, gx, gy, weight) = got
    if kind == "view":
        return image, ft, None
    *ds, dsigma = torch.autograd.grad((image * dimage).sum(), screen + [sigma])
    pgrad = torch.zeros((3, n, 4), dtype=torch.float64, device=aos.device)
    pgrad[0, idx, 0:2], pgrad[0, idx, 2:4] = ds[0], ds[1][:, 0:2]
    pgrad[1, idx, 0], pgrad[1, idx, 1], pgrad[1, idx, 2:4] = ds[1][:, 2], ds[2], ds[3][:, 0:2]
    pgrad[2, idx, 0] = ds[3][:, 2]
    for k, v in enumerate(((dsigma * gx).abs(), (dsigma * gy).abs(), weight)):
        pgrad[2, :, 1 + k] = torch.zeros(n, dtype=torch.float64, device=aos.device).index_add_(0, idx[g], v)
    del dsigma, g, sigma, gx, gy, weight
    grads, = torch.autograd.grad([mean2d, conic, opacity, color], aos, ds)
    if kind == "host":
        return image.detach(), grads
    return image.detach(), ft.detach(), None, pgrad, _planes64(grads)


def _exact_loss(case, state):
    w, h = case["width"], case["height"]
    x = state["pred"].double().reshape(h, w, 3).permute(2, 0, 1)[:, None].requires_grad_(True)
    y = state["target"].double().reshape(h, w, 3).permute(2, 0, 1)[:, None]
    if case["u8"]:
        y = y / 255.0
    k = torch.exp(-(torch.arange(11, dtype=torch.float64, device=x.device) - 5) ** 2 / 4.5)
    k = k / k.sum()

    def blur(v):
        v = torch.nn.functional.conv2d(v, k[None, None, None, :], padding=(0, 5))
        return torch.nn.functional.conv2d(v, k[None, None, :, None], padding=(5, 0))

    mx, my = blur(x), blur(y)
    sx, sy, sxy = blur(x * x) - mx * mx, blur(y * y) - my * my, blur(x * y) - mx * my
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    ssim = ((2 * mx * my + c1) * (2 * sxy + c2) / ((mx * mx + my * my + c1) * (sx + sy + c2))).mean()
    lam = _f32(0.2)
    loss = (1 - lam) * (x - y).abs().mean() + lam * (1 - ssim)
    grad, = torch.autograd.grad(loss, x)
    mse = ((x.detach().clamp(0, 1) - y.clamp(0, 1)) ** 2).mean()
    out = torch.stack([loss.detach(), ssim.detach(), -10 * torch.log10(mse)])
    return out, grad[:, 0].permute(1, 2, 0).reshape(-1)


def _exact_policy(state):
    t = state["theta"].double().requires_grad_(True)
    at, layers = 0, []
    for a, b in ((16, 64), (64, 64), (64, 3)):
        layers.append((t[at:at + a * b].reshape(a, b), t[at + a * b:at + a * b + b]))
        at += a * b + b

    def logits(v):
        for i, (m, b) in enumerate(layers):
            v = v @ m + b
            if i < 2:
                v = v * torch.sigmoid(v)
        return v

    with torch.no_grad():
        prob = torch.softmax(logits(state["x"].double()), 1)
    rw = state["rw"].double()
    nll = torch.nn.functional.cross_entropy(logits(state["rx"].double()), state["ry"].long(), reduction="none")
    grad, = torch.autograd.grad((rw * nll).sum() / rw.sum(), t)
    return prob, grad
