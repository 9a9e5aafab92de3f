"""The compositor with and without each buffer it can do without -- packed entry records, contributor bits, packed
gradient rows -- on the same inputs: channel counts, tile sizes, filters, dense and packed entries whose number is no
multiple of a warp.

Images come from the same staged values (bit-equal).  Gradients are sums of the same terms, added by atomics in another
order: 1e-6 relative.  Only anisotropic_bilinear without contributor bits integrates its footprints again, in a kernel
compiled apart: there an alpha's last place, 2^-24, over the smallest transmittance, 1e-4 (test_gpu_groups).
"""
import numpy as np
import pytest
import torch

from tests._util import rel_l2, to_np
from textured_gaussians_b200 import _backend as B
from textured_gaussians_b200 import scenes
from textured_gaussians_b200.cuda import (
    fully_fused_projection_2dgs,
    isect_offset_encode,
    isect_tiles,
    make_texture_storage,
)
from textured_gaussians_b200.cuda import _wrapper

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
W, H, N = 90, 70, 437


def T(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to(DEV, torch.float32)


def _run(D, tile=16, textured=True, filtering="bilinear", packed=False, store="fp32", absgrad=False, only_colors=False):
    """Images, statistics and gradients of one call (through the autograd function itself: five channels too)."""
    s = scenes.tiny(seed=12, N=N, R=8)
    K = T(scenes.intrinsics(80, W / 2, H / 2)[None])
    p = fully_fused_projection_2dgs(T(s.means), T(s.quats), T(s.scales), T(s.viewmats), K, W, H, packed=packed)
    kw, gid = {}, None
    if packed:
        cam, gid = p[:2]
        kw = dict(packed=True, n_cameras=1, camera_ids=cam, gaussian_ids=gid)
        p = p[2:]
    radii, means2d, depths, M, normals = p
    tw, th = -(-W // tile), -(-H // tile)
    _, ids, flat = isect_tiles(means2d, radii, depths, tile, tw, th, **kw)
    off = isect_offset_encode(ids, 1, tw, th)
    g = torch.Generator(device=DEV).manual_seed(4)
    rnd = lambda *shape: torch.rand(*shape, generator=g, device=DEV)  # noqa: E731
    table = rnd(N, D)
    colors, opac = (table[gid], T(s.opacities)[gid]) if packed else (table[None], T(s.opacities)[None])
    tex = T(s.textures)
    leaves = [x.detach().contiguous().requires_grad_() for x in (means2d, M, colors, opac, normals, tex)]
    dens = torch.zeros_like(means2d, requires_grad=True)
    held, scales = make_texture_storage(leaves[5].detach(), store) if textured else (None, None)
    layout = dict(batch_depth=32) if filtering == "anisotropic_bilinear" else None
    out = _wrapper._RasterizeToPixelsTextured.apply(
        leaves[0], leaves[1], leaves[2], leaves[3], leaves[5], leaves[4], dens, None, None, held, scales, 3.0, 3.0, W,
        H, tile, off, flat, absgrad, 0.0, 1.0, _wrapper._FILTER_ADJOINT[filtering] if textured else B.TG_ADJ_REFERENCE,
        not textured, gid, N, layout, True, 3 if filtering == "mipmapped2" else 0,
        _wrapper._FILTER_CODE.get(filtering, B.TG_FILTER_BILINEAR) if textured else B.TG_FILTER_BILINEAR)
    n_up = 1 if only_colors else 5
    ups = [2 * rnd(*o.shape) - 1 for o in out[:5]][:n_up]
    want = leaves[:5] + [dens] + ([leaves[5]] if textured else [])
    grads = list(torch.autograd.grad(out[:n_up], want, ups))
    return list(out), grads + ([leaves[0].absgrad] if absgrad else [])


def _compare(monkeypatch, patch, tol=1e-6, **case):
    images, grads = _run(**case)
    patch(monkeypatch)
    images2, grads2 = _run(**case)
    for k in (0, 1, 2, 3, 4, 6):
        assert torch.equal(images[k], images2[k]), k
    assert any(g.abs().max() > 0 for g in grads)
    for k, (a, b) in enumerate(zip(grads, grads2)):
        assert (b.abs().max() == 0) if a.abs().max() == 0 else rel_l2(to_np(b), to_np(a)) <= tol, k


def _with_records(mp):
    mp.setattr(_wrapper, "_entry_records", lambda means2d, flatten_ids: torch.full(
        (means2d.numel() // 2, 20), float("nan"), device=DEV))


def _without_bits(mp):
    mp.setattr(_wrapper, "CONTRIB_MASK_BYTES", 0)


def _without_rows(mp):
    make = torch.empty

    def empty(shape, *a, **kw):
        if tuple(shape)[-1:] == (24,):
            raise torch.cuda.OutOfMemoryError("the gradient rows do not fit")
        return make(shape, *a, **kw)

    mp.setattr(torch, "empty", empty)


PATCHES = {"records": _with_records, "no bits": _without_bits, "no rows": _without_rows}


@pytest.mark.parametrize("patch", list(PATCHES))
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("textured", [False, True])
@pytest.mark.parametrize("D", [1, 2, 3, 4, 5])
def test_channels(monkeypatch, patch, packed, textured, D):
    _compare(monkeypatch, PATCHES[patch], D=D, textured=textured, packed=packed)


@pytest.mark.parametrize("patch", list(PATCHES))
@pytest.mark.parametrize("filtering", ["bilinear", "bilinear_bwd2", "bilinear_exact", "mipmapped2",
                                       "anisotropic_bilinear"])
@pytest.mark.parametrize("only_colors", [False, True])
def test_filters(monkeypatch, patch, filtering, only_colors):
    again = patch == "no bits" and filtering == "anisotropic_bilinear"
    _compare(monkeypatch, PATCHES[patch], tol=2.0 ** -24 / 1e-4 if again else 1e-6, D=3, filtering=filtering, tile=8,
             only_colors=only_colors, absgrad=not only_colors)


@pytest.mark.parametrize("patch", list(PATCHES))
@pytest.mark.parametrize("tile", [8, 32])
@pytest.mark.parametrize("store", ["bf16", "fp8"])
def test_tiles_and_storage(monkeypatch, patch, tile, store):
    _compare(monkeypatch, PATCHES[patch], D=4, tile=tile, store=store)
