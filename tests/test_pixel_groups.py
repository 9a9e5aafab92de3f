"""CPU check of the compositor's per-group splat lists against the oracle.

Every 4x2 pixel group of the compositor visits only the splats whose image can
reach it (group_mask in textured_gaussians_b200/csrc/raster_common.cuh: the
cull box's UV square as a quadrilateral, cut into bands of two pixel rows,
united with the disk around the projected centre).  This test restates those
masks in FP64 for single random splats and requires every pixel that the FP32
oracle lights to lie in a listed group.
"""
import math

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_cull_box import cull_box

TILE = 16


def group_mask(xy, opac, M, textured, tex_square, g_weight, X0, Y0, side):
    """[side/2, side/4] booleans: the groups (two rows, four columns each) that the splat can reach."""
    nb, nc = side // 2, side // 4
    box = cull_box(xy, opac, M, textured, 3.0, 3.0, g_weight, tex_square)
    if box is None:
        return np.ones((nb, nc), bool)
    K = ((1 / (255 * opac) - 0.998 + g_weight) / g_weight if textured else 1 / (255 * opac)) * 0.999
    sig1 = 0.0 if K >= 1 else -math.log(K) * 1.001 + 1e-3
    rs, rd = math.sqrt(2 * sig1), math.sqrt(sig1)
    h = max(rs, 3.0) if textured and tex_square else rs
    q = [M @ np.array([u, v, 1.0]) for u, v in ((-h, -h), (h, -h), (h, h), (-h, h))]
    zs = [abs(c[2]) for c in q]
    q = [(c[0] / c[2], c[1] / c[2]) for c in q]
    mg = 0.25 + 1e-3 * (box[2] - box[0] + box[3] - box[1]) + 2e-6 * (max(abs(box[0]), abs(box[2]))
                                                                     + max(abs(box[1]), abs(box[3])))
    out = np.zeros((nb, nc), bool)
    for k in range(nb):
        ya = Y0 + 0.5 + 2 * k
        yb = ya + 1
        lo, hi = math.inf, -math.inf
        if min(zs) > 0.1 * max(zs):
            for i in range(4):
                (xa, y0), (xb, y1) = q[i], q[(i + 1) % 4]
                e0, e1 = min(y0, y1), max(y0, y1)
                if e1 < ya - mg or e0 > yb + mg:
                    continue
                sl = (xb - xa) / (y1 - y0) if y1 != y0 else 0.0
                for y in (ya - mg, yb + mg):
                    x = xa + (min(max(y, e0), e1) - y0) * sl
                    lo, hi = min(lo, x), max(hi, x)
            lo, hi = lo - mg, hi + mg
            d = max(ya - xy[1], xy[1] - yb, 0.0)
            if d <= rd + mg:
                w = math.sqrt((rd + mg) ** 2 - d * d)
                lo, hi = min(lo, xy[0] - w), max(hi, xy[0] + w)
        elif not (box[3] < ya or box[1] > yb):
            lo, hi = box[0], box[2]
        for c in range(nc):
            x0 = X0 + 4 * c + 0.5
            out[k, c] = hi >= x0 and lo <= x0 + 3
    return out


@pytest.mark.parametrize("form", ["plain", "bilinear", "mipmapped2", "anisotropic_bilinear"])
@pytest.mark.parametrize("W,H", [(64, 64), (2048, 16)])
def test_no_lit_pixel_outside_its_groups(form, W, H):
    rng = np.random.default_rng({"plain": 11, "bilinear": 12, "mipmapped2": 13, "anisotropic_bilinear": 14}[form] + W)
    f = 50.0 * W / 64
    lit_total = listed = box_listed = 0
    for it in range(30):
        z = rng.uniform(1.0, 4.0)
        means = np.array([[rng.uniform(-0.6, 0.6) * z, rng.uniform(-0.6, 0.6) * z * H / W, z]])
        quats = rng.normal(size=(1, 4))
        s = np.exp(rng.normal(-2.3 if W == H else -5.0, 1.2, size=2))  # thin and oblique ones among them
        K = np.array([[[f, 0, W / 2], [0, f, H / 2], [0, 0, 1]]])
        radii, m2d, _, M, nrm = O.project_fwd(means, quats / np.linalg.norm(quats), np.array([[s[0], s[1], s[1]]]),
                                              np.eye(4)[None], K, W, H)
        if radii[0, 0] <= 0:
            continue
        opac = float(rng.choice([1.0 / 254, 0.02, 0.3, 0.95]))
        g_weight = float(rng.choice([1.0, 0.6, 0.15]))
        tex = tex_arg = None
        if form != "plain":
            tex = rng.uniform(0, 1, size=(1, 8, 8, 4))
            tex[..., 3] *= rng.choice([1.0, 3.0])
            tex_arg = O.generate_mipmap(tex) if form == "mipmapped2" else tex
        tw, th = W // TILE, H // TILE
        offsets = np.arange(tw * th, dtype=np.int32).reshape(1, th, tw)  # the one splat listed in every tile
        o = O.raster_fwd(m2d, M, np.full((1, 1, 3), 0.5), np.array([[opac]]), nrm, tex_arg, offsets,
                         np.zeros(tw * th, np.int32), W, H, TILE, g_weight=g_weight,
                         mip_levels=3 if form == "mipmapped2" else 0, aniso=form == "anisotropic_bilinear",
                         dtype=np.float32)
        lit = o.alphas[0, :, :, 0] > 0
        lit_total += int(lit.sum())
        args = (m2d[0, 0].astype(float), opac, M[0, 0].astype(float), form != "plain", form != "anisotropic_bilinear",
                g_weight)
        for side in (8, 16):
            for Y0 in range(0, H, side):
                for X0 in range(0, W, side):
                    m = group_mask(*args, X0, Y0, side).repeat(2, 0).repeat(4, 1)
                    assert not (lit[Y0:Y0 + side, X0:X0 + side] & ~m).any(), (form, it, side, X0, Y0)
                    if side == 8:
                        listed += int(m.sum())
        box = cull_box(*args[:4], 3.0, 3.0, g_weight, tex_square=args[4])
        box_listed += W * H if box is None else int((min(max(box[2], 0), W) - min(max(box[0], 0), W))
                                                    * (min(max(box[3], 0), H) - min(max(box[1], 0), H)))
    assert lit_total > 0 and listed < 1.1 * box_listed  # groups round up to 4x2 pixels, yet list about what the box does
