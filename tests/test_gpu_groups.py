"""GPU parity of the compositor's pixel-group walk, both directions, against the FP64 oracle at the sizes where
it can go wrong: images of one pixel up to a few tiles with ragged right and bottom edges, every tile size (a
32x32 tile runs as four squares), batches shorter and longer than a tile's list, every channel count.

Tolerances: images as in test_gpu_parity, 1e-5 absolute (a stated share of discrete flips apart).  Gradients of
images this small can come from a few saturated pixels alone, whose final transmittance the adjoint takes from the
stored FP32 alpha: its last place, 2^-24, over the smallest transmittance the forward leaves, 1e-4, bounds the
relative error of every term of such a pixel by 6e-4, which is the relative L2 tolerance here.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests._util import assert_close, rel_l2, to_np
from textured_gaussians_b200 import scenes
from textured_gaussians_b200.cuda import (
    fully_fused_projection_2dgs,
    isect_offset_encode,
    isect_tiles,
    rasterize_to_pixels_2dgs,
    rasterize_to_pixels_textured_gaussians,
)

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
GRAD_TOL = 2.0 ** -24 / 1e-4
SIZES = [(1, 1), (7, 9), (33, 17), (65, 31), (130, 70)]


def T(x, dtype=torch.float32):
    return torch.from_numpy(np.ascontiguousarray(x)).to(DEV, dtype)


@pytest.mark.parametrize("depth", [0, 32, 1024])
@pytest.mark.parametrize("tile", [8, 16, 32])
@pytest.mark.parametrize("W,H", SIZES)
def test_textured_matches_oracle(W, H, tile, depth):
    _check(W, H, tile, depth, 3, True)


@pytest.mark.parametrize("D", [1, 2, 3, 4])
@pytest.mark.parametrize("textured", [False, True])
@pytest.mark.parametrize("tile", [8, 16, 32])
def test_channels_match_oracle(D, textured, tile):
    _check(65, 31, tile, 0, D, textured)


def _check(W, H, tile, depth, D, textured):
    s = scenes.tiny(seed=W + 7 * H, N=700, width=W, height=H)
    rng = np.random.default_rng(W * H + D)
    Ks = np.stack([scenes.intrinsics(0.9 * max(W, H, 16), W / 2, H / 2)]).astype(np.float32)
    radii, means2d, depths, M, normals = fully_fused_projection_2dgs(T(s.means), T(s.quats), T(s.scales),
                                                                     T(s.viewmats), T(Ks), W, H)
    tw, th = -(-W // tile), -(-H // tile)
    _, ids, flat = isect_tiles(means2d, radii, depths, tile, tw, th)
    off = isect_offset_encode(ids, 1, tw, th)
    colors = rng.uniform(0, 1, size=(1, 700, D)).astype(np.float32)
    opac = s.opacities[None]
    leaves = [means2d.detach().requires_grad_(), M.detach().requires_grad_(), T(colors).requires_grad_(),
              T(opac).requires_grad_(), normals.detach().requires_grad_()]
    dens = torch.zeros_like(means2d, requires_grad=True)
    tex = T(s.textures).requires_grad_()
    kw = dict(batch_depth=depth)
    if textured:
        out = rasterize_to_pixels_textured_gaussians(leaves[0], leaves[1], leaves[2], leaves[3], tex, 3.0, 3.0,
                                                     leaves[4], dens, W, H, tile, off, flat, **kw)
    else:
        out = rasterize_to_pixels_2dgs(leaves[0], leaves[1], leaves[2], leaves[3], leaves[4], dens, W, H, tile, off,
                                       flat, **kw)
    f64 = dict(dtype=np.float64)
    args = (to_np(means2d), to_np(M), colors, opac, to_np(normals), s.textures if textured else None,
            off.cpu().numpy(), flat.cpu().numpy(), W, H, tile)
    o = O.raster_fwd(*args, **f64)
    for k, ref in enumerate((o.colors, o.alphas, o.normals, o.distort)):
        assert_close(to_np(out[k]), ref, 1e-5, 1e-5, 2e-3 if W * H > 500 else 0.0, name=f"output {k}")
    assert_close(to_np(out[5]), o.contrib_sum, 1e-4, 1e-5, 2e-2, name="contrib_sum")
    up = [rng.normal(size=x.shape).astype(np.float32) for x in (o.colors, o.alphas, o.normals, o.distort)]
    up[3] *= 1e-2
    for only_colors in (False, True):
        ups = [u if k < 2 or not only_colors else np.zeros_like(u) for k, u in enumerate(up)]
        got = torch.autograd.grad(out[:2] if only_colors else out[:4], leaves + ([tex] if textured else []) + [dens],
                                  [T(u) for u in (ups[:2] if only_colors else ups)], retain_graph=True,
                                  allow_unused=True)
        r = O.raster_bwd(*args, o, *[u.astype(np.float64) for u in ups], np.zeros_like(o.median), **f64)
        refs = [r.v_means2d, r.v_M, r.v_colors, r.v_opacities, r.v_normals] + ([r.v_textures] if textured else []) + \
            [r.v_densify]
        for k, (a, b) in enumerate(zip(got, refs)):
            if np.abs(b).max() > 0:
                assert rel_l2(to_np(a), np.asarray(b).reshape(to_np(a).shape)) < GRAD_TOL, (k, only_colors)
            else:
                assert a is None or np.abs(to_np(a)).max() == 0, (k, only_colors)
