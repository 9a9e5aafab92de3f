"""The anisotropic_bilinear forward's three ways of taking squares -- a CTA of eight warps for the longest, four
squares to a CTA for the rest, and, from 18,944 squares on, the other filters' kernel -- against one another: the same
pixels rendered as part of a large image (the last way) and of smaller ones (the first two), lists longer than a step
and than a word among them.

The same sums in the same order, compiled apart: at most a rounding of 2^-24 of each accumulated value apart, so
1e-6 for images of values below about 3; the flips this can cause at the 1/255 and 1e-4 cuts may touch a pixel in a
thousand.
"""
import numpy as np
import pytest
import torch

from tests._util import assert_close, rel_l2, to_np
from textured_gaussians_b200 import scenes
from textured_gaussians_b200.rendering import rasterization_textured_gaussians

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _render(s, W, H, tile, n, depth):
    T = lambda x: torch.tensor(np.asarray(x, np.float32)[:n], device=DEV)  # noqa: E731
    leaves = [T(x).requires_grad_() for x in (s.means, s.quats, s.scales, s.opacities, s.colors, s.textures)]
    K = torch.tensor(scenes.intrinsics(900, 400, 400)[None], dtype=torch.float32, device=DEV)
    out = rasterization_textured_gaussians(*leaves, torch.tensor(s.viewmats, device=DEV), K, W, H, sh_degree=0,
                                           tile_size=tile, filtering="anisotropic_bilinear", batch_depth=depth)
    return leaves, out


@pytest.mark.parametrize("tile,depth", [(8, 0), (8, 64), (16, 32)])
@pytest.mark.parametrize("n", [3, 700])
def test_large_and_small_images_agree(tile, depth, n):
    s = scenes.tiny(seed=21, N=700, R=16)
    s.means[:300] *= 0.05  # a pile-up in the middle: lists of several hundred
    big_leaves, big = _render(s, 1600, 800, tile, n, depth)
    small_leaves, small = _render(s, 800, 800, tile, n, depth)
    for k in (0, 1, 2, 5):
        assert_close(to_np(big[k][:, :, :800]), to_np(small[k]), 1e-6, 1e-6, 1e-3, name=f"output {k}")
    up = torch.randn_like(small[0])
    gb = torch.autograd.grad(big[0][:, :, :800], big_leaves, up)
    gs = torch.autograd.grad(small[0], small_leaves, up)
    for k, (a, b) in enumerate(zip(gb, gs)):
        assert rel_l2(to_np(a), to_np(b)) < 2.0 ** -24 / 1e-4, k  # (test_gpu_groups: the stored alpha's last place)


@pytest.mark.parametrize("tile,depth", [(8, 608), (8, 640), (8, 1024), (16, 640), (16, 1024)])
def test_deep_batches_agree_with_shallow_ones(tile, depth):
    """Batches of up to 1024 splats, of which four squares' do not fit one CTA's shared memory together above 608."""
    s = scenes.tiny(seed=22, N=1500, R=16)
    s.means[:1200] *= 0.02  # lists longer than a batch
    deep_leaves, deep = _render(s, 800, 800, tile, 1500, depth)
    leaves, ref = _render(s, 800, 800, tile, 1500, 32)
    for k in (0, 1, 2, 5):
        assert_close(to_np(deep[k]), to_np(ref[k]), 1e-6, 1e-6, 1e-3, name=f"output {k}")
    up = torch.randn_like(ref[0])
    for k, (a, b) in enumerate(zip(torch.autograd.grad(deep[0], deep_leaves, up),
                                   torch.autograd.grad(ref[0], leaves, up))):
        assert rel_l2(to_np(a), to_np(b)) < 2.0 ** -24 / 1e-4, k
