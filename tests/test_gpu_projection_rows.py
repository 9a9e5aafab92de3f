"""The dense projection's warp-staged rows against the packed projection, which writes and reads them one thread per
row: Gaussian counts around a warp's 32 and a CTA's 64 / 128, every SH degree, with rows longer than the degree
needs, one and several cameras (odd camera strides misalign the staged vectors).

Forward outputs are the same device function's: bit-equal.  Gradients sum the same per-entry terms in another order
(cameras in registers here, atomics there): 4 FP32 roundings of 2^-24 per camera and value, so 1e-6 relative L2.
"""
import pytest
import torch

from tests._util import rel_l2, to_np
from textured_gaussians_b200 import scenes
from textured_gaussians_b200.cuda import fully_fused_projection_2dgs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("degree,K", [(None, 0), (0, 1), (0, 4), (1, 4), (2, 9), (2, 16), (3, 16), (4, 25)])
@pytest.mark.parametrize("N", [1, 31, 33, 64, 127, 129, 300])
@pytest.mark.parametrize("C", [1, 3])
def test_dense_matches_packed(N, C, degree, K):
    s = scenes.tiny(seed=N + 7 * C, N=N, n_cams=C)
    g = torch.Generator(device=DEV).manual_seed(N)
    leaves = [torch.tensor(x, device=DEV).requires_grad_() for x in (s.means, s.quats, s.scales)]
    sh = None
    if degree is not None:
        sh = torch.randn(N, K, 3, generator=g, device=DEV).mul_(0.5).requires_grad_()
    V, Ks = torch.tensor(s.viewmats, device=DEV), torch.tensor(s.Ks, device=DEV)
    kw = dict(sh_coeffs=sh, sh_degree=degree)
    dense = fully_fused_projection_2dgs(*leaves, V, Ks, s.width, s.height, **kw)
    packed = fully_fused_projection_2dgs(*leaves, V, Ks, s.width, s.height, packed=True, **kw)
    cam, gid = packed[0], packed[1]
    assert torch.equal(torch.stack([cam, gid], 1), (dense[0] > 0).nonzero())
    for d, p in zip(dense, packed[2:]):
        assert torch.equal(d[cam, gid], p)
    if len(gid) == 0:
        return
    ups = [torch.randn(p.shape, generator=g, device=DEV) for p in packed[3:]]
    wrt = leaves + ([] if sh is None else [sh])
    gp = torch.autograd.grad(packed[3:], wrt, ups)
    full = []
    for d, u in zip(dense[1:], ups):
        f = torch.zeros_like(d)
        f[cam, gid] = u
        full.append(f)
    gd = torch.autograd.grad(dense[1:], wrt, full)
    for k, (a, b) in enumerate(zip(gd, gp)):
        assert rel_l2(to_np(a), to_np(b)) < 1e-6, k
