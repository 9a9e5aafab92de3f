"""GPU parity of the depth-image pass (expected depth and normals from depth) with the tensor expressions in FP64, both
directions, at sizes around its 32x8 tiles.

Tolerances.  Focal length 50 and depths around 2, so central differences are about 4 / 50 = 0.08 long; a point up to 4
long carries at most six roundings (6 * 4 * 2^-24 = 1.4e-6), a difference twice that, a tangent's direction
2.9e-6 / 0.08 = 3.6e-5 and a normal, from two tangents, 7.2e-5: 1e-4.  Gradients are products of two such quantities
with an upstream up to 1, summed over four neighbours: 5e-4 of the largest.
"""
import pytest
import torch

from textured_gaussians_b200.cuda._wrapper import depth_image
from textured_gaussians_b200.utils import depth_image_expression, depth_to_normal

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("W,H", [(2, 2), (3, 3), (32, 8), (33, 9), (34, 10), (31, 65), (130, 7)])
@pytest.mark.parametrize("C,D,expected,median", [(1, 4, True, False), (3, 4, False, False), (2, 4, True, True),
                                                 (2, 1, True, False)])
def test_depth_image(W, H, C, D, expected, median):
    g = torch.Generator().manual_seed(W * 100 + H)
    rnd = lambda *s: torch.rand(*s, generator=g)  # noqa: E731
    al = 0.25 + 0.75 * rnd(C, H, W, 1)
    y, x = torch.meshgrid(torch.arange(H) / 9.0, torch.arange(W) / 7.0, indexing="ij")
    z = (2.0 + 0.2 * torch.sin(x + y))[None, :, :, None].expand(C, H, W, 1)
    colors = torch.cat([rnd(C, H, W, D - 1), z * al if expected else z], -1)
    med = z + 0.01 * rnd(C, H, W, 1) if median else None
    c2w = torch.eye(4).repeat(C, 1, 1)
    c2w[:, :3, :3] = torch.linalg.qr(torch.randn(C, 3, 3, generator=g))[0]
    c2w[:, :3, 3] = 0.5 * rnd(C, 3)
    Ks = torch.tensor([[50.0, 0, W / 2], [0, 50.0, H / 2], [0, 0, 1]]).repeat(C, 1, 1)
    with_n = D == 4
    ups = [2 * rnd(C, H, W, D) - 1, 2 * rnd(C, H, W, 3) - 1]

    def run(fused, dt):
        t = [None if v is None else v.to(DEV, dt).requires_grad_() for v in (colors, al, med)]
        cam = [c2w.to(DEV, dt), Ks.to(DEV, dt)]
        if fused:
            out, n = depth_image(t[0], t[1] if expected else None, t[2], *(cam if with_n else ()))
        else:
            out = torch.cat([t[0][..., :-1], t[0][..., -1:] / t[1].clamp(min=1e-10)], -1) if expected else None
            d = t[2] if median else (out if expected else t[0])[..., -1:]
            n = depth_to_normal(d, *cam) if with_n else None
        loss = sum((o * u.to(DEV, dt)).sum() for o, u in zip((out, n), ups) if o is not None)
        leaves = [v for v in t if v is not None]
        return [out, n], torch.autograd.grad(loss, leaves, allow_unused=True)

    got, ref = run(True, torch.float32), run(False, torch.float64)
    for a, b, tol in zip(got[0], ref[0], (1e-6 * 4, 1e-4)):
        assert (a is None) == (b is None)
        if a is not None:
            assert a.shape == b.shape and (a.double() - b).abs().max() < tol
    for a, b in zip(got[1], ref[1]):
        assert (a is None or a.abs().max() == 0) if b is None else (
            (a.double() - b).abs().max() <= 5e-4 * b.abs().max())


@pytest.mark.parametrize("expected,median", [(True, False), (False, False), (True, True)])
def test_second_derivatives(expected, median):
    """A derivative of the gradient: taken of the same FP32 expressions on either side, so alike but for the order in
    which a few shares of a gradient are added (a handful of roundings of 2^-24: 1e-5 of the largest is ample)."""
    W, H, D = 40, 21, 4
    g = torch.Generator().manual_seed(3)
    rnd = lambda *s: torch.rand(*s, generator=g).to(DEV)  # noqa: E731
    colors, al, med = rnd(2, H, W, D) + 1, 0.25 + 0.75 * rnd(2, H, W, 1), rnd(2, H, W, 1) + 1
    cam = (torch.eye(4, device=DEV).repeat(2, 1, 1),
           torch.tensor([[50.0, 0, W / 2], [0, 50.0, H / 2], [0, 0, 1]], device=DEV).repeat(2, 1, 1))
    ups = [rnd(2, H, W, D), rnd(2, H, W, 3)]
    res = []
    for fn in (depth_image, depth_image_expression):
        t = [v.clone().requires_grad_() for v in ((colors, al) if expected else (colors,)) + ((med,) if median else ())]
        out, n = fn(t[0], t[1] if expected else None, t[-1] if median else None, *cam)
        loss = sum((o * u).sum() for o, u in zip((out, n), ups) if o is not None)
        first = torch.autograd.grad(loss, t, create_graph=True)
        assert all(f.requires_grad for f in first if f.abs().max() > 0)
        second = torch.autograd.grad(sum((f * f).sum() for f in first), t)
        res.append((first, second))
    for a, b in zip(res[0][0] + res[0][1], res[1][0] + res[1][1]):
        assert (a - b).abs().max() <= 1e-5 * b.abs().max()
    assert all(s.abs().max() > 0 for s in res[0][1])
