"""The calls this package is used for, as measurable cases: renders, training steps and the steps around them.

Every case is a dict of plain values.  ``prepare`` draws its inputs on the GPU (the value distributions of
``textured_gaussians_b200.scenes``: uniform cubes of small splats seen from 4 units, or a 64-component mixture seen
from 25), ``run`` makes one pass through the public entry points and ``exact`` gives the same outputs in 64-bit torch
where that is affordable.  Paths:

  render      forward only, no gradients (viewer, evaluation)
  train       forward, image loss, gradients of every parameter (one optimisation step's renderer work)
  batch       the same over several scenes and views of uneven size in one call
  projection  the projection op alone, both directions, SH colours fused
  isect       tile intersection, key sort and tile offsets
  adam        the optimiser step on the textures of the visible splats, plus densification statistics
"""
from __future__ import annotations

import math

import numpy as np
import torch

import textured_gaussians_b200.scenes as scenes
from textured_gaussians_b200.batch import ViewTable, rasterization_textured_gaussians_batch
from textured_gaussians_b200.cuda._wrapper import (densify_stats, fully_fused_projection_2dgs, isect_offset_encode,
                                                   isect_tiles, make_texture_storage)
from textured_gaussians_b200.optimizers import SelectiveAdam
from textured_gaussians_b200.rendering import rasterization_2dgs, rasterization_textured_gaussians

DEV = "cuda"

# scene: "cube" (scales exp(N(-4, 0.5)), camera at 4, white-noise textures) or "mixture" (scales exp(N(-3.5, 0.6)),
# camera at 25, smooth textures).  tex 0: plain 2DGS.  depth 0: the default batch depth.
_BASE = {"path": "train", "scene": "mixture", "splats": 100000, "tex": 32, "storage": "fp32", "filter": "bilinear",
         "views": 1, "width": 800, "height": 600, "tile": 16, "depth": 0, "sh": 0, "mode": "RGB", "packed": False,
         "dist": False}


def _case(name=None, **kw):
    c = {**_BASE, **kw}
    return c if name is None else {"name": name, **c}


def listed():
    return [
        # a small preview frame: 10k splats with 8x8 textures, 200x200, the drop-in defaults; launch latency counts
        _case("render_small", path="render", scene="cube", splats=10000, tex=8, width=200, height=200),
        # the smallest training step (a unit-scale fit): 2k splats, 128x128
        _case("train_small", scene="cube", splats=2000, tex=16, width=128, height=128),
        # plain 2DGS training with depth, distortion loss and packed entries (the geometry stage before texturing)
        _case("train_2dgs", scene="cube", splats=150000, tex=0, width=800, height=800, sh=3, mode="RGB+ED",
              packed=True, dist=True),
        # the drop-in textured step of an object scene: FP32 50x50 textures, one 800x800 view, SH degree 3, tile 16
        _case("train_views", scene="cube", splats=100000, tex=50, width=800, height=800, sh=3),
        # interactive viewing of a trained scene: BF16 storage, one odd-sized 1297x840 frame
        _case("render_view", path="render", splats=500000, storage="bf16", width=1297, height=840, tile=8, depth=64),
        # the largest training step: 1M splats, four 1600x1200 views in one call, BF16 storage
        _case("train_mixture", splats=1000000, storage="bf16", views=4, width=1600, height=1200, tile=8, depth=64),
        # the mip-mapped filter at an ordinary size
        _case("train_mipmapped2", splats=150000, storage="bf16", filter="mipmapped2", width=1600, height=1200, tile=8),
        # the footprint-integrating filter at an ordinary size
        _case("train_anisotropic", splats=60000, filter="anisotropic_bilinear", width=800, height=600, tile=8),
        # two scenes, six views of uneven sizes, one call
        _case("train_batch", path="batch", splats=200000, storage="bf16", views=6, width=1297, height=840, tile=8,
              depth=64),
        # what every step starts with: 1M splats into four cameras with SH degree 3, and its adjoint
        _case("projection", path="projection", splats=1000000, views=4, sh=3, width=1600, height=1200),
        # the tile lists of an ordinary frame: intersection, 64-bit key sort, offsets
        _case("intersections", path="isect", splats=500000, views=2, width=1600, height=1200, tile=16),
        # the update after a step: selective Adam on FP32 textures with their BF16 copy, and the densification statistics
        _case("update", path="adam", splats=200000, storage="bf16", views=2, width=800, height=600),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["render", "train", "train", "train", "plain", "filter", "batch", "projection", "isect", "adam"])
    w, h = _log_int(rng, 120, 1600), _log_int(rng, 100, 1200)
    views = rng.choice([1, 1, 2, 3])
    tile = rng.choice([8, 16])
    if path in ("render", "train"):
        cube = rng.random() < 0.4
        storage = "fp32" if cube else rng.choice(["fp32", "bf16", "bf16", "fp16", "fp8"])
        return _case(path=path, scene="cube" if cube else "mixture", splats=_log_int(rng, 2000, 60000 if cube else 300000),
                     tex=rng.choice([8, 16, 21, 50] if cube else [16, 32, 32, 27]), storage=storage, views=views,
                     width=w, height=h, tile=tile, depth=rng.choice([0, 0, 64, 128]), sh=rng.choice([0, 1, 3]),
                     mode=rng.choice(["RGB", "RGB", "RGB+ED"]), packed=rng.random() < 0.3)
    if path == "plain":
        mode = rng.choice(["RGB", "RGB+D", "RGB+ED"])
        return _case(scene="cube", splats=_log_int(rng, 2000, 200000), tex=0, views=views, width=w, height=h, tile=tile,
                     sh=rng.choice([0, 2, 3]), mode=mode, packed=rng.random() < 0.5,
                     dist=mode != "RGB" and rng.random() < 0.5)
    if path == "filter":
        f = rng.choice(["mipmapped2", "anisotropic_bilinear"])
        most = 80000 if f == "mipmapped2" else 25000  # a smaller image has larger footprints to integrate
        return _case(splats=_log_int(rng, 5000, most), tex=rng.choice([16, 32]), storage=rng.choice(["fp32", "bf16"]),
                     filter=f, width=min(w, 1000), height=min(h, 800), tile=tile)
    if path == "batch":
        return _case(path="batch", splats=_log_int(rng, 10000, 200000), storage=rng.choice(["fp32", "bf16"]),
                     views=rng.choice([3, 4, 5, 7]), width=min(w, 1297), height=min(h, 840), tile=tile,
                     sh=rng.choice([0, 3]))
    if path == "projection":
        return _case(path="projection", splats=_log_int(rng, 20000, 1000000), views=rng.choice([1, 2, 4, 5]),
                     sh=rng.choice([0, 1, 2, 3]), width=w, height=h)
    if path == "isect":
        return _case(path="isect", splats=_log_int(rng, 5000, 800000), views=views, width=w, height=h, tile=tile)
    return _case(path="adam", splats=_log_int(rng, 2000, 200000), tex=rng.choice([8, 16, 25, 32]),
                 storage=rng.choice(["fp32", "bf16", "fp16"]), views=views, width=w, height=h)


# ------------------------------------------------------------------------------------------------ inputs
def _uniform(g, *shape):
    return torch.rand(shape, generator=g, device=DEV)


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device=DEV)


def _smooth_textures(g, n, r):
    """0.5 + a 4x4 block of low cosine frequencies, clamped to [0, 1]."""
    x = torch.arange(r, device=DEV, dtype=torch.float32)
    basis = torch.cos(math.pi * (2 * x[:, None] + 1) * torch.arange(4, device=DEV)[None] / (2 * r))
    out = torch.empty((n, r, r, 4), device=DEV)
    for s in range(0, n, 65536):
        a = 0.3 * _normal(g, min(65536, n - s), 4, 4, 4)
        out[s:s + 65536] = torch.einsum("yv,xu,nvuc->nyxc", basis, basis, a).add_(0.5).clamp_(0.0, 1.0)
    return out


def _splats(c, g):
    """means, quats, scales, opacities, colours (SH coefficients) and textures of the case's scene."""
    n, k = c["splats"], (c["sh"] + 1) ** 2
    if c["scene"] == "cube":
        means, mu, sd, op = 2 * _uniform(g, n, 3) - 1, -4.0, 0.5, 0.0
    else:
        u = _normal(g, 64, 3)
        centres = u / u.norm(dim=1, keepdim=True) * 10.0 * _uniform(g, 64, 1) ** (1.0 / 3.0)
        means = centres[torch.randint(0, 64, (n,), generator=g, device=DEV)] + 0.5 * _normal(g, n, 3)
        mu, sd, op = -3.5, 0.6, 0.5
    ls = mu + sd * _normal(g, n, 2)
    q = _normal(g, n, 4)
    s = {"means": means, "quats": q / q.norm(dim=1, keepdim=True), "scales": torch.cat([ls, ls[:, 1:]], 1).exp(),
         "opacities": torch.sigmoid(op + _normal(g, n)),
         "colors": torch.cat([_uniform(g, n, 1, 3), 0.05 * _normal(g, n, k - 1, 3)], 1)}
    if c["tex"] and c["path"] not in ("projection", "isect"):
        r = c["tex"]
        s["textures"] = _uniform(g, n, r, r, 4) if c["scene"] == "cube" else _smooth_textures(g, n, r)
    return s


def _sizes(c):
    """Image size of each view: all the same, or (batch) cycling through smaller and odd ones."""
    w, h = c["width"], c["height"]
    if c["path"] != "batch":
        return [(w, h)] * c["views"]
    return [[(w, h), (w // 2, h // 2), (w // 3 + 1, h // 3)][i % 3] for i in range(c["views"])]


def _cameras(c):
    radius, focal = (4.0, 1.1) if c["scene"] == "cube" else (25.0, 0.75)
    dirs = scenes.fibonacci_dirs(max(c["views"], 1) + 1)
    V = np.stack([scenes.look_at(radius * d) for d in dirs[:c["views"]]])
    K = np.stack([scenes.intrinsics(focal * w, w / 2, h / 2) for w, h in _sizes(c)])
    return (torch.tensor(V, dtype=torch.float32, device=DEV), torch.tensor(K, dtype=torch.float32, device=DEV))


def _channels(c):
    return {"RGB": 3, "D": 1, "ED": 1}.get(c["mode"], 4)


def prepare(case, seed):
    c = case
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    s = _splats(c, g)
    s["viewmats"], s["Ks"] = _cameras(c)
    s["case"] = c
    n, C = c["splats"], c["views"]
    if c["path"] in ("render", "train", "batch"):
        s["background"] = _uniform(g, C, 3) if c["mode"] == "RGB" and c["filter"] == "bilinear" else None
        if c["tex"] and c["storage"] != "fp32":
            s["storage"], s["tex_scales"] = make_texture_storage(s["textures"], c["storage"])
        if c["path"] != "render":
            s["targets"] = [_uniform(g, h, w, _channels(c)) for w, h in _sizes(c)]
            if c["path"] == "train":
                s["targets"] = torch.stack(s["targets"])
            for k in ("means", "quats", "scales", "opacities", "colors", "textures"):
                if k in s:
                    s[k].requires_grad_(True)
        if c["path"] == "batch":
            s["offsets"] = [0, n // 4, n]
            s["view_scenes"] = [i % 2 for i in range(C)]
            ws, hs = zip(*_sizes(c))
            s["views"] = ViewTable(ws, hs, c["tile"], torch.device(DEV))
    elif c["path"] == "projection":
        for k in ("means", "quats", "scales", "colors"):
            s[k].requires_grad_(True)
        s["upstream"] = [_normal(g, C, n, 2), _normal(g, C, n), _normal(g, C, n, 3, 3), _normal(g, C, n, 3),
                         _normal(g, C, n, 3)]
    elif c["path"] == "isect":
        with torch.no_grad():
            p = fully_fused_projection_2dgs(s["means"], s["quats"], s["scales"], s["viewmats"], s["Ks"], c["width"],
                                            c["height"])
        # the lists' length depends on the scene: they are kept in buffers of a size that covers every seed
        room = 16 * C * n
        s = {"case": c, "radii": p[0], "means2d": p[1], "depths": p[2],
             "ids": torch.zeros(room, dtype=torch.int64, device=DEV),
             "flatten": torch.zeros(room, dtype=torch.int32, device=DEV)}
    else:  # adam: a scene's textures after a backward, with the splats' visibility
        tex = s["textures"]
        s["visible"] = _uniform(g, n) < 0.7
        s["grad"] = 1e-3 * _normal(g, *tex.shape)
        s["shadow"] = tex.to({"bf16": torch.bfloat16, "fp16": torch.float16}[c["storage"]]) if c["storage"] != "fp32" \
            else None
        param = torch.nn.Parameter(tex)
        s["opt"] = SelectiveAdam([{"params": [param], "lr": 2.5e-3}], eps=1e-15, betas=(0.9, 0.999),
                                 shadows={} if s["shadow"] is None else {param: s["shadow"]})
        s["textures"] = param
        s["radii"] = (60 * _uniform(g, C, n) - 10).int().clamp_(min=0)
        s["grads2d"] = 1e-4 * _normal(g, C, n, 2)
        s["stats"] = [torch.zeros(n, device=DEV) for _ in range(3)]
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _leaves(s):
    return [s[k] for k in ("means", "quats", "scales", "opacities", "colors", "textures") if k in s]


def _render(s, c):
    kw = dict(sh_degree=c["sh"], packed=c["packed"], tile_size=c["tile"], backgrounds=s["background"],
              render_mode=c["mode"], batch_depth=c["depth"])
    if c["tex"]:
        kw.update(filtering=c["filter"], texture_storage=s.get("storage"), texture_scales=s.get("tex_scales"))
        return rasterization_textured_gaussians(s["means"], s["quats"], s["scales"], s["opacities"], s["colors"],
                                                s["textures"], s["viewmats"], s["Ks"], c["width"], c["height"], **kw)
    return rasterization_2dgs(s["means"], s["quats"], s["scales"], s["opacities"], s["colors"], s["viewmats"], s["Ks"],
                              c["width"], c["height"], distloss=c["dist"], **kw)


def run(state):
    s, c = state, state["case"]
    if c["path"] == "render":
        with torch.no_grad():
            colors, alphas, normals, from_depth, distort, median, _, _, _ = _render(s, c)
        return {"colors": colors, "alphas": alphas, "normals": normals, "depth_normals": from_depth,
                "distort": distort, "median": median}
    if c["path"] == "train":
        colors, alphas, normals, from_depth, distort, median, csum, _, meta = _render(s, c)
        loss = (colors - s["targets"]).square().mean()
        if c["dist"]:
            loss = loss + 0.1 * distort.mean() + 0.05 * (normals - 0.5).square().mean()
        grads = torch.autograd.grad(loss, _leaves(s) + [meta["gradient_2dgs"]])
        out = {"colors": colors, "alphas": alphas, "normals": normals, "depth_normals": from_depth,
               "distort": distort, "median": median, "contrib": csum}
        out = {k: None if v is None else v.detach() for k, v in out.items()}
        return {**out, "grads": list(grads[:-1]), "densify": grads[-1]}
    if c["path"] == "batch":
        ws, hs = zip(*_sizes(c))
        colors, alphas, normals, _, _, _, csum, _, meta = rasterization_textured_gaussians_batch(
            s["means"], s["quats"], s["scales"], s["opacities"], s["colors"], s["textures"], s["offsets"],
            s["viewmats"], s["Ks"], ws, hs, s["view_scenes"], sh_degree=c["sh"], tile_size=c["tile"],
            backgrounds=s["background"], batch_depth=c["depth"], texture_storage=s.get("storage"),
            view_table=s["views"])
        loss = sum((a - t).square().mean() for a, t in zip(colors, s["targets"]))
        grads = torch.autograd.grad(loss, _leaves(s))
        return {"colors": [x.detach() for x in colors], "alphas": [x.detach() for x in alphas], "contrib": csum,
                "grads": list(grads)}
    if c["path"] == "projection":
        radii, means2d, depths, rt, normals, cols = fully_fused_projection_2dgs(
            s["means"], s["quats"], s["scales"], s["viewmats"], s["Ks"], c["width"], c["height"],
            sh_coeffs=s["colors"], sh_degree=c["sh"])
        outs = [means2d, depths, rt, normals, cols]
        grads = torch.autograd.grad(outs, [s["means"], s["quats"], s["scales"], s["colors"]], s["upstream"])
        return {"radii": radii, "outs": [o.detach() for o in outs], "grads": list(grads)}
    if c["path"] == "isect":
        tw, th = -(-c["width"] // c["tile"]), -(-c["height"] // c["tile"])
        counts, ids, flat = isect_tiles(s["means2d"], s["radii"], s["depths"], c["tile"], tw, th)
        s["ids"][:len(ids)].copy_(ids)
        s["flatten"][:len(flat)].copy_(flat)
        return {"counts": counts, "ids": s["ids"], "flatten": s["flatten"],
                "offsets": isect_offset_encode(ids, c["views"], tw, th)}
    s["textures"].grad = s["grad"]
    s["opt"].step(s["visible"])
    densify_stats(s["grads2d"], s["radii"], c["width"], c["height"], c["views"], *s["stats"])
    st = s["opt"].state[s["textures"]]
    out = {"textures": s["textures"].detach(), "exp_avg": st["exp_avg"], "exp_avg_sq": st["exp_avg_sq"],
           "stats": list(s["stats"])}
    return out if s["shadow"] is None else {**out, "shadow": s["shadow"]}


# ------------------------------------------------------------------------------------------------ work
def _footprint_pixels(c):
    """Mean pixels inside a splat's 6-sigma square, turned at random to the camera (half its face-on area)."""
    dist, foc, mu, sd = (4.0, 1.1, -4.0, 0.5) if c["scene"] == "cube" else (25.0, 0.75, -3.5, 0.6)
    px = math.exp(mu + sd * sd) * foc / dist
    return sum(18.0 * (px * w) ** 2 for w, _ in _sizes(c))


def work(case):
    c = case
    n, C, k = c["splats"], c["views"], (c["sh"] + 1) ** 2
    per_splat = 4 * (3 + 4 + 3 + 1 + 3 * k)
    pixels = sum(w * h for w, h in _sizes(c))
    texel = {"fp32": 16, "bf16": 8, "fp16": 8, "fp8": 4}[c["storage"]]
    if c["path"] in ("render", "train", "batch"):
        t = c["tex"] ** 2
        b = n * (per_splat + t * texel) + 4 * pixels * (_channels(c) + 6)
        f = n * _footprint_pixels(c) * 80
        if c["path"] != "render":
            b += n * (per_splat + 16 * t) + 8 * pixels * _channels(c)
            f *= 3.5
        return {"bytes": b, "flops": f}
    if c["path"] == "projection":
        return {"bytes": n * 2 * (per_splat - 4) + C * n * 4 * (19 + 18 + 3), "flops": C * n * (700 + 60 * k)}
    if c["path"] == "isect":
        cover = 4.0 + 9.0 * (0.036 * 0.75 * c["width"] / 25.0 / c["tile"]) ** 2  # tiles a splat meets, roughly
        return {"bytes": C * n * (20 + 12 * cover), "flops": C * n * cover * 8}
    t = 4 * c["tex"] ** 2
    return {"bytes": 0.7 * n * t * (16 + 12 + (0 if c["storage"] == "fp32" else 2)) + n * (24 + 12 * C),
            "flops": 0.7 * n * t * 12}


# ------------------------------------------------------------------------------------------------ 64-bit values
def _rotation(q):
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    c0 = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y)], 1)
    c1 = torch.stack([2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x)], 1)
    c2 = torch.stack([2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)], 1)
    return c0, c1, c2


def _sh(degree, d, coeffs):
    """Real spherical harmonics (degree <= 3) of directions d [N,3] with coefficients [N,K,3]."""
    x, y, z = (d / d.norm(dim=1, keepdim=True)).unbind(1)
    one = torch.ones_like(x)
    b = [0.5 * math.sqrt(1 / math.pi) * one]
    if degree >= 1:
        k = math.sqrt(3 / (4 * math.pi))
        b += [-k * y, k * z, -k * x]
    if degree >= 2:
        k = math.sqrt(15 / (4 * math.pi))
        b += [k * x * y, -k * y * z, math.sqrt(5 / (16 * math.pi)) * (3 * z * z - 1), -k * x * z,
              0.5 * k * (x * x - y * y)]
    if degree >= 3:
        k1, k2, k3 = math.sqrt(35 / (32 * math.pi)), math.sqrt(105 / (4 * math.pi)), math.sqrt(21 / (32 * math.pi))
        b += [-k1 * y * (3 * x * x - y * y), k2 * x * y * z, -k3 * y * (5 * z * z - 1),
              math.sqrt(7 / (16 * math.pi)) * z * (5 * z * z - 3), -k3 * x * (5 * z * z - 1),
              0.5 * k2 * z * (x * x - y * y), -k1 * x * (x * x - 3 * y * y)]
    return (torch.stack(b, 1)[:, :, None] * coeffs[:, :len(b)]).sum(1)


def _project(p, V, K, width, height, degree):
    """One camera: visible mask, radius and the per-splat means2d, depth, ray transform, normal, colour with their
    graph; the gradient of means2d reaches the ray transform through its diagonal terms alone (the package's
    default adjoint)."""
    R, t = V[:3, :3], V[:3, 3]
    mc = p["means"] @ R.T + t
    c0, c1, c2 = (c @ R.T for c in _rotation(p["quats"]))
    WH = torch.stack([p["scales"][:, :1] * c0, p["scales"][:, 1:2] * c1, mc], 2)
    M = K @ WH
    m = M.detach()
    sgn = torch.tensor([1.0, 1.0, -1.0], dtype=torch.float64, device=DEV)
    f = 1.0 / (m[:, 2] ** 2 * sgn).sum(1)
    xy = (m[:, :2] * m[:, 2:] * sgn).sum(2) * f[:, None]
    hh = xy ** 2 - (m[:, :2] ** 2 * sgn).sum(2) * f[:, None]
    radius = torch.ceil(3 * hh.amax(1).clamp(min=1e-4).sqrt())
    vis = ((mc[:, 2] >= 0.01) & (mc[:, 2] <= 1e10) & (xy[:, 0] + radius > 0) & (xy[:, 0] - radius < width)
           & (xy[:, 1] + radius > 0) & (xy[:, 1] - radius < height)).detach()
    # value xy, gradient d xy_j / d M[j] = sgn f M[2] and d xy_j / d M[2] = sgn M[j] (f -+ 2 f^2 M[2]^2)
    g2 = sgn * (f[:, None] - sgn * 2 * f[:, None] ** 2 * m[:, 2] ** 2)
    sur = (M[:, :2] * (sgn * f[:, None] * m[:, 2])[:, None]).sum(2) + (M[:, 2:] * (m[:, :2] * g2[:, None])).sum(2)
    means2d = xy + sur - sur.detach()
    mult = torch.where((-c2 * mc).sum(1) > 0, 1.0, -1.0).detach()
    centre = -torch.linalg.solve(R, t)
    col = (_sh(degree, p["means"] - centre, p["colors"]) + 0.5).clamp_min(0.0)
    return vis, radius, means2d, mc[:, 2], M, mult[:, None] * c2, col


def _tiles(c, w, h, vis, radius, xy, depth):
    """Depth-sorted splat lists of the view's tiles: (flat ids, tile starts, tile ends)."""
    ts, tw, th = c["tile"], -(-w // c["tile"]), -(-h // c["tile"])
    idx = vis.nonzero()[:, 0]
    idx = idx[torch.argsort(depth[idx], stable=True)]
    r, x, y = radius[idx] / ts, xy[idx, 0] / ts, xy[idx, 1] / ts
    x0, x1 = torch.floor(x - r).clamp(0, tw).long(), torch.ceil(x + r).clamp(0, tw).long()
    y0, y1 = torch.floor(y - r).clamp(0, th).long(), torch.ceil(y + r).clamp(0, th).long()
    cnt = (x1 - x0) * (y1 - y0)
    rep = torch.repeat_interleave(torch.arange(len(idx), device=DEV), cnt)
    k = torch.arange(len(rep), device=DEV) - (torch.cumsum(cnt, 0) - cnt)[rep]
    tile = (y0[rep] + k // (x1 - x0)[rep]) * tw + x0[rep] + k % (x1 - x0)[rep]
    order = torch.argsort(tile, stable=True)
    bounds = torch.searchsorted(tile[order], torch.arange(tw * th + 1, device=DEV))
    return idx[rep[order]], bounds[:-1], bounds[1:]


def _composite(c, ids, live, px, py, e, tex, bg):
    """Tiles [B] with lists ids [B,L] and pixel centres px, py [B,P]: colours, alphas, normals, distortion, median,
    per-pair alphas of the contributors.  e: per-splat M, xy, opacity, colour, normal; tex [N,R,R,4] or None."""
    M = e["M"][ids][:, None]  # [B,1,L,3,3]
    hu = px[..., None, None] * M[..., 2, :] - M[..., 0, :]
    hv = py[..., None, None] * M[..., 2, :] - M[..., 1, :]
    z = torch.linalg.cross(hu, hv)
    zz = torch.where(z[..., 2] == 0, 1.0, z[..., 2])
    sx, sy = z[..., 0] / zz, z[..., 1] / zz
    g3 = sx * sx + sy * sy
    d = e["xy"][ids][:, None] - torch.stack([px, py], -1)[:, :, None]
    g2 = 2.0 * (d * d).sum(-1)
    kern = torch.exp(-0.5 * torch.where(g3 <= g2, g3, g2))
    op = e["opacity"][ids][:, None]
    cols = e["colors"][ids][:, None].expand(*sx.shape, -1)
    if tex is None:
        raw = op * kern
    else:
        ux, uy = sx.detach(), sy.detach()
        inside = (ux.abs() <= 3.0) & (uy.abs() <= 3.0)
        R = tex.shape[1]
        u, v = (((t + 3.0) / 6.0 * (R - 1)).clamp(0, R - 1) for t in (ux, uy))
        ul, vl = u.floor().long(), v.floor().long()
        uh, vh = u.ceil().long(), v.ceil().long()
        wu, wv = u - ul, v - vl
        flat = tex.view(-1, 4)
        base = ids[:, None] * (R * R)
        smp = 0.0
        for vv, uu, w in ((vl, ul, (1 - wu) * (1 - wv)), (vl, uh, wu * (1 - wv)), (vh, ul, (1 - wu) * wv),
                          (vh, uh, wu * wv)):
            smp = smp + w[..., None] * flat[base + vv * R + uu].double()
        smp = torch.where(inside[..., None], smp, 0.0)
        raw = op * (kern - 0.002) * torch.where(inside, smp[..., 3], 1.0)
        cols = cols + torch.nn.functional.pad(smp, (0, cols.shape[-1]))[..., :cols.shape[-1]]
    alpha = raw.clamp(max=0.999)
    ok = live[:, None] & (z[..., 2] != 0) & (alpha >= 1.0 / 255.0)
    alpha = torch.where(ok, alpha, 0.0)
    ok = ok & (torch.cumprod(1 - alpha.detach(), -1) > 1e-4)
    alpha = torch.where(ok, alpha, 0.0)
    T = torch.cumprod(1 - alpha, -1)
    before = torch.cat([torch.ones_like(T[..., :1]), T[..., :-1]], -1)
    wgt = alpha * before
    rgb = (wgt[..., None] * cols).sum(2)
    left = T[..., -1]
    if bg is not None:
        rgb = rgb + left[..., None] * bg
    nrm = (wgt[..., None] * e["normals"][ids][:, None]).sum(2)
    m = e["colors"][ids][:, None, :, -1]
    wm = wgt * m
    dist = 2 * (wm * (1 - before) - wgt * (torch.cumsum(wm, -1) - wm)).sum(-1)
    at = (ok & (before.detach() > 0.5)).long() * torch.arange(1, ids.shape[1] + 1, device=DEV)
    last = at.amax(-1)
    med = torch.where(last > 0, torch.gather(m.expand_as(wgt), 2, (last - 1).clamp(min=0)[..., None])[..., 0], 0.0)
    return rgb, 1 - left, nrm, dist, med, alpha


_PAIRS = 1.0e9  # (pixel, listed splat) pairs of a case up to which its 64-bit values are computed


def _view_exact(c, s, p, tex, vtex, view, w, h, bg, target, n_loss, acc, normals_world):
    """One view's outputs in 64 bits, and its gradients added to acc (None: forward only); None if too many pairs."""
    V, K = s["viewmats"][view].double(), s["Ks"][view].double()
    vis, radius, xy, depth, M, nrm, col = _project(p, V, K, w, h, c["sh"])
    cols = {"RGB": col, "D": depth[:, None], "ED": depth[:, None]}.get(c["mode"])
    cols = torch.cat([col, depth[:, None]], 1) if cols is None else cols
    ts, tw, th = c["tile"], -(-w // c["tile"]), -(-h // c["tile"])
    ids, lo, hi = _tiles(c, w, h, vis, radius, xy.detach(), depth.detach())
    if float((hi - lo).sum()) * ts * ts * c["views"] > _PAIRS:
        return None
    leaf = {"M": M, "xy": xy, "opacity": p["opacities"], "colors": cols, "normals": nrm}
    grad = acc is not None
    e = {k: v.detach().requires_grad_(grad) for k, v in leaf.items()}
    sums = {k: torch.zeros_like(v) for k, v in e.items()}
    D = cols.shape[1]
    out = {k: torch.zeros((h, w) + t, dtype=torch.float64, device=DEV)
           for k, t in (("colors", (D,)), ("alphas", (1,)), ("normals", (3,)), ("distort", (1,)), ("median", (1,)))}
    contrib = torch.zeros(c["splats"], dtype=torch.float64, device=DEV)
    off = torch.arange(ts * ts, device=DEV)
    order = torch.argsort(hi - lo, descending=True)
    ends = (hi - lo)[order].tolist()
    rot = torch.linalg.inv(V)[:3, :3] if normals_world else None
    at = 0
    while at < len(ends):
        L = max(1, ends[at])
        B = max(1, min(len(ends) - at, int(4.0e6 // (L * ts * ts)) or 1))
        tiles = order[at:at + B]
        at += B
        pos = lo[tiles][:, None] + torch.arange(L, device=DEV)
        live = pos < hi[tiles][:, None]
        tid = torch.where(live, ids[pos.clamp(max=max(len(ids) - 1, 0))] if len(ids) else 0, 0)
        X = (tiles % tw)[:, None] * ts + off % ts
        Y = (tiles // tw)[:, None] * ts + off // ts
        keep = (X < w) & (Y < h)
        with torch.set_grad_enabled(grad):
            if vtex is not None:  # texture gradients of the lists' splats
                uniq, inv = torch.unique(tid, return_inverse=True)
                tx = tex[uniq].double().requires_grad_(True)
                sub = {k: v[uniq] for k, v in e.items()}
                rgb, al, nr, ds, md, alpha = _composite(c, inv, live, X + 0.5, Y + 0.5, sub, tx, bg)
            else:
                rgb, al, nr, ds, md, alpha = _composite(c, tid, live, X + 0.5, Y + 0.5, e, tex, bg)
            if "ED" in c["mode"]:
                rgb = torch.cat([rgb[..., :-1], rgb[..., -1:] / al.clamp(min=1e-10)[..., None]], -1)
            nw = nr if rot is None else nr @ rot.T
            yx = (Y[keep], X[keep])
            for k, t in (("colors", rgb), ("alphas", al[..., None]), ("normals", nw), ("distort", ds[..., None]),
                         ("median", md[..., None])):
                out[k][yx] = t.detach()[keep]
            contrib.index_add_(0, tid.reshape(-1), (alpha.detach() * keep[..., None]).sum(1).reshape(-1))
            if grad:
                loss = (rgb[keep] - target[yx].double()).square().sum() / (n_loss * D)
                if c["dist"]:
                    loss = loss + 0.1 * ds[keep].sum() / n_loss + 0.05 * (nw[keep] - 0.5).square().sum() / (3 * n_loss)
                wrt = list(e.values()) + ([tx] if vtex is not None else [])
                got = torch.autograd.grad(loss, wrt, allow_unused=True)
                for k, v in zip(e, got):
                    if v is not None:
                        sums[k] += v
                if vtex is not None and got[-1] is not None:
                    vtex.index_add_(0, uniq, got[-1])
    out["contrib"] = contrib
    if grad:
        out["densify"] = torch.where(vis[:, None], sums["M"][:, :2, 2] * M.detach()[:, 2:, 2], 0.0)
        got = torch.autograd.grad([leaf[k] for k in leaf], list(p.values()), [sums[k] for k in leaf],
                                  allow_unused=True)
        for k, v in zip(p, got):
            if v is not None:
                acc[k] += v
    return out


def _exact_render(c, seed):
    grad = c["path"] != "render"
    if c["filter"] != "bilinear":
        return None  # the footprint filters have no short 64-bit form here
    if c["splats"] * c["tex"] ** 2 > 3e8:
        return None
    s = prepare(c, seed)
    tex = vtex = None
    if c["tex"]:
        tex = s["textures"].detach() if c["storage"] == "fp32" else s["storage"]
        if s.get("tex_scales") is not None:
            tex = tex.float() * s["tex_scales"][:, None, None, None]
        elif tex.dtype != torch.float32:
            tex = tex.float()
        vtex = torch.zeros(tex.shape, dtype=torch.float64, device=DEV) if grad else None
    names = ("means", "quats", "scales", "opacities", "colors")
    P = {k: s[k].detach().double().requires_grad_(grad) for k in names}
    acc = {k: torch.zeros_like(v) for k, v in P.items()} if grad else None
    sizes, outs = _sizes(c), []
    for v, (w, h) in enumerate(sizes):
        a, b = (0, c["splats"])
        if c["path"] == "batch":
            a, b = s["offsets"][s["view_scenes"][v]:][:2]
        sub = {k: t[a:b] for k, t in P.items()}
        with torch.set_grad_enabled(grad):
            cut = {k: t.detach().requires_grad_(grad) for k, t in sub.items()}
            part = {k: t[a:b] for k, t in acc.items()} if grad else None
            bg = None if s["background"] is None else s["background"][v].double()
            n_loss = w * h * (1 if c["path"] == "batch" else c["views"])
            got = _view_exact({**c, "splats": b - a}, s, cut, None if tex is None else tex[a:b],
                              None if vtex is None else vtex[a:b], v, w, h, bg,
                              s["targets"][v] if grad else None, n_loss, part, c["path"] != "batch")
        if got is None:
            return None
        got["range"] = (a, b)
        outs.append(got)
    contrib = torch.zeros(c["splats"], dtype=torch.float64, device=DEV)
    for o in outs:
        contrib[o["range"][0]:o["range"][1]] += o["contrib"]
    grads = None if not grad else [acc[k] for k in names] + ([vtex] if vtex is not None else [])
    if c["path"] == "batch":
        return {"colors": [o["colors"] for o in outs], "alphas": [o["alphas"] for o in outs], "contrib": contrib,
                "grads": grads}
    img = {k: torch.stack([o[k] for o in outs]) for k in ("colors", "alphas", "normals", "distort", "median")}
    img["depth_normals"] = None
    if not grad:
        return img
    return {**img, "contrib": contrib, "grads": grads,
            "densify": None if c["packed"] else torch.stack([o["densify"] for o in outs])}


def _exact_projection(c, seed):
    s = prepare(c, seed)
    p = {k: s[k].detach().double().requires_grad_(True) for k in ("means", "quats", "scales", "colors")}
    outs, acc = [], {k: torch.zeros_like(v) for k, v in p.items()}
    for v in range(c["views"]):
        vis, _, xy, depth, M, nrm, col = _project(p, s["viewmats"][v].double(), s["Ks"][v].double(), c["width"],
                                                  c["height"], c["sh"])
        view = [torch.where(vis.reshape(-1, *[1] * (t.dim() - 1)), t, f)
                for t, f in ((xy, 0.0), (depth, 0.0), (M, 0.0), (nrm, 0.0), (col, 0.5))]
        got = torch.autograd.grad(view, list(p.values()), [u[v].double() for u in s["upstream"]])
        for k, t in zip(p, got):
            acc[k] += t
        outs.append([t.detach() for t in view])
    return {"outs": [torch.stack(t) for t in zip(*outs)], "grads": list(acc.values()), "radii": None}


def _exact_update(c, seed):
    s = prepare(c, seed)
    on = s["visible"][:, None, None, None]
    g = s["grad"].double()
    m, v = torch.where(on, 0.1 * g, 0.0), torch.where(on, (1 - 0.999) * g * g, 0.0)
    t = s["textures"].detach().double()
    t = torch.where(on, t - 2.5e-3 * m / (v.sqrt() + 1e-15), t)
    seen = s["radii"] > 0
    scale = torch.tensor([c["width"] / 2 * c["views"], c["height"] / 2 * c["views"]], dtype=torch.float64, device=DEV)
    r = s["radii"].double() / max(c["width"], c["height"])
    stats = [torch.where(seen, (s["grads2d"].double() * scale).norm(dim=-1), 0.0).sum(0), seen.sum(0).double(),
             torch.where(seen, r, 0.0).amax(0)]
    out = {"textures": t, "exp_avg": m, "exp_avg_sq": v, "stats": stats}
    return out if s["shadow"] is None else {**out, "shadow": t}


def exact(case, seed):
    c = case
    if c["path"] == "isect":
        return None  # whole numbers only
    if c["path"] == "projection":
        return _exact_projection(c, seed)
    if c["path"] == "adam":
        return _exact_update(c, seed)
    return _exact_render(c, seed)
