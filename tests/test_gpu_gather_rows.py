"""The packed layout's gather of per-Gaussian inputs: a row's gradient is summed over its entries in FP32, whatever the
table's type.  Tolerance: FP32 sums of 256 terms (256 roundings of 2^-24, 1.5e-5, at worst), rounded once to the
table's type: half a unit of its last place, 2^-11 (FP16), 2^-8 (BF16), relative."""
import pytest
import torch

from textured_gaussians_b200.cuda._wrapper import gather_rows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype,tol", [(torch.float16, 2.0 ** -11), (torch.bfloat16, 2.0 ** -8), (torch.float32, 0.0)])
@pytest.mark.parametrize("shape", [(500,), (500, 3)])
def test_gradients_are_summed_in_fp32(dtype, tol, shape):
    g = torch.Generator(device=DEV).manual_seed(1)
    views, n = 256, shape[0]
    ids = torch.arange(n, device=DEV).repeat(views)
    table = torch.randn(shape, generator=g, device=DEV).to(dtype).requires_grad_()
    up = torch.rand((views * n,) + shape[1:], generator=g, device=DEV).to(dtype)
    out = gather_rows(table, ids)
    assert out.dtype == dtype and torch.equal(out, table.detach().repeat(views, *[1] * (len(shape) - 1)))
    got, = torch.autograd.grad(out, table, up)
    want = up.double().view(views, *shape).sum(0)
    assert got.dtype == dtype
    assert ((got.double() - want).abs() <= (tol + 1.5e-5) * want.abs()).all()
