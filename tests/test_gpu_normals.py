"""GPU parity of the normal-image rotation against the FP64 torch expression, both directions, at sizes around its
1024-pixel chunks and with unaligned views.

Tolerance: three FP32 products and two sums of values up to 1 and matrix entries up to 1 in magnitude, so at most
5 roundings of 2^-24 of values up to 3, plus the matrix entries' own rounding (2^-24 each, three products): 2e-6.
"""
import numpy as np
import pytest
import torch

from textured_gaussians_b200 import scenes
from textured_gaussians_b200.batch import ViewTable
from textured_gaussians_b200.cuda._wrapper import normals_to_world

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _views(C):
    return torch.tensor(np.stack([scenes.look_at(4.0 * d) for d in scenes.fibonacci_dirs(C)]), dtype=torch.float32,
                        device=DEV)


@pytest.mark.parametrize("W,H", [(1, 1), (31, 33), (32, 32), (1025, 1), (64, 50)])
@pytest.mark.parametrize("C", [1, 3])
def test_one_size(W, H, C):
    V = _views(C)
    n = (torch.rand(C, H, W, 3, device=DEV) * 2 - 1).requires_grad_()
    up = torch.rand_like(n) * 2 - 1
    out = normals_to_world(n, V)
    (g,) = torch.autograd.grad(out, n, up)
    A = torch.linalg.inv(V.double())[:, :3, :3]
    assert (out.double() - torch.einsum("cij,chwj->chwi", A, n.double())).abs().max() < 2e-6
    assert (g.double() - torch.einsum("cij,chwi->chwj", A, up.double())).abs().max() < 2e-6
    Vg = V.clone().requires_grad_()  # view matrices that need a gradient keep getting one
    normals_to_world(n, Vg).sum().backward()
    assert Vg.grad.abs().max() > 0


def test_uneven_views():
    sizes = [(33, 7), (5, 3), (64, 32), (1, 1), (130, 9)]
    V = _views(len(sizes))
    vt = ViewTable([w for w, _ in sizes], [h for _, h in sizes], 8, torch.device(DEV))
    n = (torch.rand(vt.n_pixels, 3, device=DEV) * 2 - 1).requires_grad_()
    out = normals_to_world(n, V, vt)
    (g,) = torch.autograd.grad(out, n, torch.ones_like(n))
    A = torch.linalg.inv(V.double())[:, :3, :3]
    for c, (b, k) in enumerate(zip(vt.pix_base, vt.pix_count)):
        assert (out[b:b + k].double() - n[b:b + k].double() @ A[c].T).abs().max() < 2e-6
        assert (g[b:b + k].double() - A[c].sum(0)).abs().max() < 2e-6
