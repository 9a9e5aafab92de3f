"""The sorted intersection lists (entries by depth, then camera and tile) and the compositor's tile order against
the general path -- entry-order emission and a sort of the whole 64-bit keys -- bit for bit, at the sizes where the
forms change: one entry, around the one-CTA sort's 16,384 entries / tiles, around 1024-entry emission chunks and
4096-pair sort tiles; dense, packed and uneven views; equal, negative and zero depths; culled entries.
"""
import numpy as np
import pytest
import torch

from textured_gaussians_b200.batch import ViewTable
from textured_gaussians_b200.cuda._wrapper import isect_tiles, sort_pairs, tile_order_heaviest_first
from textured_gaussians_b200.graph import SizePlan

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _bits(n):
    return int(n).bit_length()


def _entries(E, W, H, seed, depths="random", radius=40):
    g = torch.Generator(device=DEV).manual_seed(seed)
    xy = torch.rand(E, 2, generator=g, device=DEV) * torch.tensor([1.2 * W, 1.2 * H], device=DEV) - 0.1 * min(W, H)
    r = (torch.rand(E, generator=g, device=DEV) ** 4 * radius).int()  # about a third of the entries culled
    if depths == "equal":
        d = torch.full((E,), 2.5, device=DEV)
    elif depths == "signed":
        d = (torch.randint(-4, 5, (E,), generator=g, device=DEV)).float()
    else:
        d = torch.rand(E, generator=g, device=DEV) * 10 + 0.01
    return xy, r, d


def _same(a, b):
    assert all(torch.equal(x, y) for x, y in zip(a, b)), [(x.shape, y.shape) for x, y in zip(a, b)]


@pytest.mark.parametrize("depths", ["random", "equal", "signed"])
@pytest.mark.parametrize("C,N", [(1, 1), (1, 1023), (2, 513), (3, 5461), (1, 16384), (1, 16385), (4, 20011)])
def test_dense(C, N, depths):
    W, H, tile = 500, 300, 16
    tw, th = -(-W // tile), -(-H // tile)
    xy, r, d = (t.view(C, N, *t.shape[1:]) for t in _entries(C * N, W, H, C * N, depths))
    cnt, ids, flat = isect_tiles(xy, r, d, tile, tw, th)
    cnt0, ids0, flat0 = isect_tiles(xy, r, d, tile, tw, th, sort=False)
    ids0, flat0 = sort_pairs(ids0, flat0, 32 + _bits(tw * th) + _bits(C))
    _same((cnt, ids, flat), (cnt0, ids0, flat0))


@pytest.mark.parametrize("E", [1, 3000, 40000])
def test_packed_and_views(E):
    sizes = [(640, 200), (33, 65), (320, 320)]
    vt = ViewTable([w for w, _ in sizes], [h for _, h in sizes], 8, torch.device(DEV))
    xy, r, d = _entries(E, 640, 320, E, radius=90)
    cam = torch.randint(0, 3, (E,), device=DEV).sort()[0]
    gid = torch.arange(E, device=DEV)
    for view_table, tw, th in ((None, 80, 40), (vt, 0, 0)):
        kw = dict(packed=True, n_cameras=3, camera_ids=cam, gaussian_ids=gid, view_table=view_table)
        got = isect_tiles(xy, r, d, 8, tw, th, **kw)
        cnt0, ids0, flat0 = isect_tiles(xy, r, d, 8, tw, th, sort=False, **kw)
        ids0, flat0 = sort_pairs(ids0, flat0, 32 + _bits(vt.key_tiles if view_table else tw * th) + _bits(3))
        _same(got, (cnt0, ids0, flat0))


@pytest.mark.parametrize("slack", [1.5, 1.0, 0.5])
def test_capacity(slack):
    W, H, tile = 500, 300, 8
    tw, th = -(-W // tile), -(-H // tile)
    xy, r, d = (t.view(1, 30000, *t.shape[1:]) for t in _entries(30000, W, H, 5))
    cnt0, ids0, flat0 = isect_tiles(xy, r, d, tile, tw, th)
    n = ids0.numel()
    cap = int(n * slack)
    with SizePlan("capture", [cap]) as plan:
        cnt, ids, flat = isect_tiles(xy, r, d, tile, tw, th)
    assert ids.numel() == cap and torch.equal(cnt, cnt0)
    assert bool(plan.flags[0].item()) == (cap < n)
    if cap >= n:
        _same((ids[:n], flat[:n]), (ids0, flat0))
        pad = (1 << (32 + _bits(tw * th) + 1)) - 1
        assert (ids[n:] == pad).all() and (flat[n:] == 0).all()
        assert int(flat._tg_n_isects.item()) == n
    else:
        assert (ids[1:] >= ids[:-1]).all()


@pytest.mark.parametrize("n_tiles", [1, 2, 31, 1025, 16384, 16385, 70001])
@pytest.mark.parametrize("longest", [0, 1, 300, 70000])
def test_tile_order(n_tiles, longest):
    g = torch.Generator(device=DEV).manual_seed(n_tiles + longest)
    counts = (torch.rand(n_tiles, generator=g, device=DEV) ** 3 * (longest + 1)).long().clamp(max=longest)
    if n_tiles > 40000:
        counts = counts // 8  # (offsets are 32-bit)
    ends = counts.cumsum(0)
    off = (ends - counts).int()
    total = int(ends[-1])
    want = torch.argsort(-counts, stable=True).int()
    assert torch.equal(tile_order_heaviest_first(off, total), want)
    assert torch.equal(tile_order_heaviest_first(off, torch.tensor([total], device=DEV)), want)
    assert np.array_equal(np.sort(want.cpu().numpy()), np.arange(n_tiles))
