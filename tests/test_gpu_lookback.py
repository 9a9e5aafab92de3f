"""Sorted lists whose look-back waits give up (nobody takes the first 4096 pairs of a sort): the call ends, what it
writes stays in range, and the next call on the same buffers is right.  The scratch is filled with 0xff first, so that
places the broken sort leaves unwritten hold ids of no entry.
"""
import ctypes

import pytest
import torch

from textured_gaussians_b200 import _backend as B
from textured_gaussians_b200.cuda._wrapper import isect_tiles, tile_order_heaviest_first

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
W, H, TILE, E = 500, 300, 16, 40000
TW, TH = -(-W // TILE), -(-H // TILE)
KEY_BITS = (TW * TH).bit_length() + 1


def _entries():
    g = torch.Generator(device=DEV).manual_seed(9)
    xy = torch.rand(1, E, 2, generator=g, device=DEV) * torch.tensor([float(W), float(H)], device=DEV)
    radii = (torch.rand(1, E, generator=g, device=DEV) ** 4 * 30).int()
    return xy, radii, torch.rand(1, E, generator=g, device=DEV) + 0.1


class Call:
    """One tg_isect_sorted_count / _lists pair on buffers of its own."""

    def __init__(self, xy, radii, depths):
        self.inputs = (xy, radii, depths)  # (read by every call)
        self.L, self.st = B.lib(), B.stream_of(xy)
        u8 = lambda n: torch.full((n,), 0xff, dtype=torch.uint8, device=DEV)  # noqa: E731
        self.order_ws = u8(self.L.tg_isect_sorted_order_bytes(E))
        self.counts = torch.empty((1, E), dtype=torch.int32, device=DEV)
        self.n_dev = torch.empty((1,), dtype=torch.int64, device=DEV)
        self.a = B.IsectArgs(E, E, None, B.ptr(xy), B.ptr(radii), B.ptr(depths), TILE, TW, TH, 1, B.ptr(self.counts),
                             None, B.ptr(self.n_dev))
        self.count()
        self.n = int(self.n_dev.item())
        self.list_ws = u8(self.L.tg_isect_sorted_lists_bytes(self.n, KEY_BITS))
        self.ids = torch.zeros((self.n,), dtype=torch.int64, device=DEV)
        self.flat = torch.zeros((self.n,), dtype=torch.int32, device=DEV)
        self.a.isect_ids, self.a.flatten_ids = B.ptr(self.ids), B.ptr(self.flat)

    def count(self):
        B.check(self.L.tg_isect_sorted_count(ctypes.byref(self.a), B.ptr(self.order_ws), self.order_ws.numel(),
                                             self.st), "count")

    def lists(self, lost=0):
        args = [ctypes.byref(self.a), B.ptr(self.order_ws), self.n, B.ptr(self.list_ws), self.list_ws.numel()]
        fn = self.L.tg_isect_sorted_lookback_selftest if lost else self.L.tg_isect_sorted_lists
        B.check(fn(*args, *([lost] if lost else []), self.st), "lists")


@pytest.mark.parametrize("lost", [1, 2])
def test_lists_stay_in_range_and_the_next_call_is_right(lost):
    inputs = _entries()
    c = Call(*inputs)
    c.lists(lost)
    torch.cuda.synchronize()
    assert int(c.flat.min()) >= 0 and int(c.flat.max()) < E
    c.count()
    c.lists()
    _, ids, flat = isect_tiles(*inputs, TILE, TW, TH)
    assert torch.equal(c.ids, ids) and torch.equal(c.flat, flat)


@pytest.mark.parametrize("lost", [1, 2])
@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("spare", [None, 0, 5000])
def test_every_place_holds_an_entry(lost, shift, spare):
    """Also the places nothing was sorted into, whatever the buffer's alignment, with exact sizes (None) and in
    capacity mode with so many places to spare: a compositor given such lists stays within the entries."""
    c = Call(*_entries())
    if spare is not None:
        flag = torch.zeros((1,), dtype=torch.int32, device=DEV)
        c.n += spare
        c.a.capacity, c.a.overflow = c.n, B.ptr(flag)
        c.list_ws = torch.full((c.L.tg_isect_sorted_lists_bytes(c.n, KEY_BITS),), 0xff, dtype=torch.uint8, device=DEV)
        c.ids = torch.zeros((c.n,), dtype=torch.int64, device=DEV)
        c.a.isect_ids = B.ptr(c.ids)
    flat = torch.full((c.n + 4,), -1, dtype=torch.int32, device=DEV)[shift:shift + c.n]
    c.a.flatten_ids = B.ptr(flat)
    c.lists(lost)
    torch.cuda.synchronize()
    assert int(flat.min()) >= 0 and int(flat.max()) < E


def _status(c):
    return c.L.tg_isect_sorted_status(B.ptr(c.order_ws), E, B.ptr(c.list_ws), c.n, KEY_BITS, c.st)


@pytest.mark.parametrize("lost", [1, 2])
def test_lists_report_it(lost):
    inputs = _entries()
    c = Call(*inputs)
    c.lists()
    assert _status(c) == 0
    c.count()
    c.lists(lost)
    assert _status(c) == -5 and b"gave up" in c.L.tg_last_error()
    c.count()
    c.lists()
    assert _status(c) == 0
    assert torch.equal(isect_tiles(*inputs, TILE, TW, TH, check=True)[2], c.flat)


@pytest.mark.parametrize("entries", [0, 5, 16384, 16385])
def test_status_of_every_size(entries):
    """The sizes whose entries one CTA sorts keep no flag: nothing else of the scratch is taken for one."""
    args = [x[:, :entries].contiguous() for x in _entries()]
    for sort in (True, False):
        isect_tiles(*args, TILE, TW, TH, sort=sort, check=True)


@pytest.mark.parametrize("n_tiles", [1, 16384, 16385, 50000])
def test_tile_order_reports_it(n_tiles):
    off = torch.arange(n_tiles, dtype=torch.int32, device=DEV) * 3
    total = 3 * n_tiles
    want = torch.arange(n_tiles, dtype=torch.int32, device=DEV)
    assert torch.equal(tile_order_heaviest_first(off, total, check=True), want)
    L, st = B.lib(), B.stream_of(off)
    ws = torch.full((L.tg_tile_order_workspace_bytes(n_tiles),), 0xff, dtype=torch.uint8, device=DEV)
    order = torch.empty_like(off)
    rc = L.tg_tile_order_lookback_selftest(B.ptr(off), n_tiles, total, B.ptr(order), B.ptr(ws), ws.numel(), st)
    if n_tiles <= 16384:
        assert rc == -1
    else:
        assert rc == 0 and L.tg_tile_order_status(B.ptr(ws), n_tiles, st) == -5
    assert L.tg_tile_order(B.ptr(off), n_tiles, total, None, B.ptr(order), B.ptr(ws), ws.numel(), st) == 0
    assert L.tg_tile_order_status(B.ptr(ws), n_tiles, st) == 0 and torch.equal(order, want)
