"""A tile order is refused where the offsets and their device count lie on different devices, before anything is
launched (the meta device stands in for a second one: no GPU is needed to find out)."""
import pytest
import torch

from textured_gaussians_b200.cuda._wrapper import tile_order_heaviest_first


@pytest.mark.parametrize("offsets,count", [("cpu", "meta"), ("meta", "cpu")])
def test_count_on_another_device_is_refused(offsets, count):
    off = torch.zeros((4,), dtype=torch.int32, device=offsets)
    n = torch.zeros((1,), dtype=torch.int64, device=count)
    with pytest.raises(RuntimeError, match="count on"):
        tile_order_heaviest_first(off, n)


@pytest.mark.gpu
def test_host_count_for_device_offsets_is_refused():
    off = torch.zeros((4,), dtype=torch.int32, device="cuda:0")
    with pytest.raises(RuntimeError, match="count on"):
        tile_order_heaviest_first(off, torch.tensor([7]))
    assert tile_order_heaviest_first(off, torch.tensor([7], device="cuda:0")).tolist() == [3, 0, 1, 2]
