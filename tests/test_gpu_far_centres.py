"""The adjoint for large splats close to the camera, whose projected centre lies up to 1e9 pixels off the image:
gradients of ray transforms, pushed on to means, rotations and scales in FP64, against the FP64 oracle.  One splat per
view, so that every splat's error stands by itself.

Tolerance: the oracle's adjoint in FP32 sums the pairs' nine products themselves and rounds each operation once; the
GPU's divisions and exponentials are good to two units of the last place where the oracle's are to half a one, four
times its error.  So the median over the splats may be 4 times the FP32 oracle's, and the largest, a maximum of a few
dozen such errors on either side, twice that.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from tests._util import to_np
from tests.test_gpu_parity import _near_degenerate_splats
from textured_gaussians_b200.batch import ViewTable
from textured_gaussians_b200.cuda import (
    fully_fused_projection_2dgs,
    isect_offset_encode,
    isect_tiles,
    rasterize_to_pixels_2dgs,
    rasterize_to_pixels_textured_gaussians,
)
from textured_gaussians_b200.cuda._wrapper import isect_offset_encode_views

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
W, H, TILE = 160, 120, 16


def T(x):
    return torch.from_numpy(np.ascontiguousarray(x)).to(DEV, torch.float32)


def _parameter_gradients(p, radii, M, v_M):
    """Gradients of each splat's mean, rotation and scales ([n, 10], FP64) from those of its ray transform."""
    out = []
    zero = lambda *s: np.zeros(s)  # noqa: E731
    for i in range(len(radii)):
        g = O.project_bwd(*[x[i:i + 1] for x in p], np.eye(4)[None], _K(), radii[i].reshape(1, 1), M[i][None, None],
                          zero(1, 1, 2), zero(1, 1), zero(1, 1, 3), v_M[i].reshape(1, 1, 3, 3).astype(np.float64),
                          dtype=np.float64)
        out.append(np.concatenate([a.ravel() for a in g]))
    return np.stack(out)


def _K():
    return np.array([[[120, 0, W / 2], [0, 120, H / 2], [0, 0, 1]]], np.float32)


@pytest.mark.parametrize("views", [False, True])
@pytest.mark.parametrize("textured,adjoint", [(False, "bilinear"), (True, "bilinear"), (True, "bilinear_exact")])
def test_gradients_keep_their_digits(textured, adjoint, views):
    p = _near_degenerate_splats(600, seed=5)
    radii, means2d, depths, M, normals = fully_fused_projection_2dgs(*map(T, p), T(np.eye(4)[None]), T(_K()), W, H)
    far = (means2d[0] - torch.tensor([W / 2, H / 2], device=DEV)).abs().amax(1)
    keep = torch.nonzero((radii[0] > 0) & (far > 4 * W))[:96, 0]
    p = [x[keep.cpu().numpy()] for x in p]
    radii, means2d, depths, M, normals = (x[0, keep][:, None].contiguous() for x in (radii, means2d, depths, M, normals))
    n = len(keep)
    assert n >= 48 and far[keep].max() > 1e6
    tw, th = -(-W // TILE), -(-H // TILE)
    _, ids, flat = isect_tiles(means2d, radii, depths, TILE, tw, th)
    off = isect_offset_encode(ids, n, tw, th)
    rng = np.random.default_rng(0)
    colors, opac = rng.uniform(0, 1, (n, 1, 3)).astype(np.float32), np.full((n, 1), 0.7, np.float32)
    tex = rng.uniform(0.3, 1, (1, 8, 8, 4)).astype(np.float32)
    up = [rng.normal(size=(n, H, W, k)).astype(np.float32) for k in (3, 1)]
    leaf = M.detach().clone().requires_grad_()
    dens = torch.zeros_like(means2d)
    args = [means2d, leaf, T(colors), T(opac)]
    kw = dict(filtering=adjoint) if textured else {}
    size = (W, H)
    if views:  # the batching form: packed entries, one row each, flat images
        vt = ViewTable([W] * n, [H] * n, TILE, torch.device(DEV))
        cam = torch.arange(n, device=DEV)
        args = [x.reshape(n, *x.shape[2:]) for x in args]
        normals, dens, size = normals.reshape(n, 3), dens.reshape(n, 2), (0, 0)
        _, ids, flat = isect_tiles(args[0], radii.reshape(n), depths.reshape(n), TILE, 0, 0, packed=True, n_cameras=n,
                                   camera_ids=cam, gaussian_ids=cam, view_table=vt)
        off_gpu = isect_offset_encode_views(ids, vt)
        kw.update(packed=True, gaussian_ids=torch.zeros_like(cam), view_table=vt)
        if not textured:
            kw["n_gaussians"] = 1
    else:
        off_gpu = off
    tail = (normals, dens, *size, TILE, off_gpu, flat)
    out = (rasterize_to_pixels_textured_gaussians(*args, T(tex), 3.0, 3.0, *tail, **kw) if textured
           else rasterize_to_pixels_2dgs(*args, *tail, **kw))
    loss = sum((o.reshape(n, H, W, -1) * T(u)).sum() for o, u in zip(out[:2], up))
    got, = torch.autograd.grad(loss, leaf)
    raster = (to_np(means2d), to_np(M), colors, opac, to_np(normals.reshape(n, 1, 3)), tex if textured else None,
              off.cpu().numpy(), np.arange(n, dtype=np.int32)[_camera(off, len(flat))], W, H, TILE)
    mode = 2 if adjoint == "bilinear_exact" else 0
    grads = {}
    for dt in (np.float64, np.float32):
        f = O.raster_fwd(*raster, dtype=dt)
        zero = [np.zeros_like(x) for x in (f.normals, f.distort, f.median)]
        grads[dt] = O.raster_bwd(*raster, f, *up, *zero, mode=mode, dtype=dt).v_M[:, 0]
    r = radii.cpu().numpy()[:, 0]
    want, base, mine = (_parameter_gradients(p, r, to_np(M)[:, 0].astype(np.float64), g)
                        for g in (grads[np.float64], grads[np.float32], to_np(got).reshape(n, 3, 3)))
    some = np.linalg.norm(want, axis=1) > 0
    assert some.sum() >= 40
    e32, err = (np.linalg.norm((g - want)[some], axis=1) / np.linalg.norm(want[some], axis=1) for g in (base, mine))
    print("FP32 oracle median %.1e max %.1e, GPU median %.1e max %.1e" % (np.median(e32), e32.max(), np.median(err),
                                                                        err.max()))
    assert np.median(err) <= 4 * np.median(e32) and err.max() <= 8 * e32.max()


def _camera(off, n_isects):
    """The view of every intersection (one splat per view: its entry)."""
    starts = off.reshape(off.shape[0], -1)[:, 0].cpu().numpy()
    return np.searchsorted(starts, np.arange(n_isects), side="right") - 1
