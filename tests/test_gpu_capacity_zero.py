"""Capacity mode with room for no intersection: what does not fit is reported, as with every other capacity."""
import pytest
import torch

from tests.test_gpu_graph import DropInStep, _check, _eager
from textured_gaussians_b200.cuda._wrapper import isect_tiles
from textured_gaussians_b200.graph import GraphedStep, SizePlan

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("sort", [True, False])
@pytest.mark.parametrize("radius", [0, 5])
@pytest.mark.parametrize("E", [3, 20000])
def test_overflow_is_raised(E, radius, sort):
    xy = torch.full((1, E, 2), 20.0, device=DEV)
    radii = torch.full((1, E), radius, dtype=torch.int32, device=DEV)
    with SizePlan("capture", [0]) as plan:
        _, ids, flat = isect_tiles(xy, radii, torch.ones(1, E, device=DEV), 16, 4, 4, sort=sort)
    assert ids.numel() == flat.numel() == 0
    assert bool(plan.flags[0].item()) == (radius > 0)


def test_graph_recorded_on_an_empty_step_reports_overflow():
    step = DropInStep()
    with torch.no_grad():
        step.leaves[0].add_(1000.0)  # out of every view
    g = GraphedStep(step, floor=0)
    assert g.sizes == [0] and g.capacities == [0]
    g.replay()
    assert not g.overflowed()
    with torch.no_grad():
        step.leaves[0].sub_(1000.0)
    g.replay()
    assert g.overflowed()
    g.recapture()
    out = tuple(t.clone() for t in g.replay())
    grads = step.grads()
    assert not g.overflowed()
    _check(out, _eager(step), grads)
