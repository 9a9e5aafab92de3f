"""What the compositor's forward keeps for its adjoint."""
import pytest
import torch

from textured_gaussians_b200 import rasterization_2dgs, rasterization_textured_gaussians, scenes
from textured_gaussians_b200.cuda import _wrapper

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _leaves(s, textured):
    names = ("means", "quats", "scales", "opacities", "colors") + (("textures",) if textured else ())
    return [torch.from_numpy(getattr(s, k)).to(DEV).requires_grad_() for k in names]


@pytest.mark.parametrize("filtering", [None, "bilinear", "anisotropic_bilinear"])
def test_renders_without_gradients_keep_nothing_for_an_adjoint(filtering, monkeypatch):
    """Under no_grad a render of parameters that require gradients makes no contributor bits and no records."""
    s = scenes.tiny(seed=3)
    L = _leaves(s, filtering is not None)
    kept = []

    def fwd_args(*a, **kw):
        kept.append(make(*a, **kw))
        return kept[-1]

    make = _wrapper._fwd_args
    monkeypatch.setattr(_wrapper, "_fwd_args", fwd_args)
    cam = (torch.from_numpy(s.viewmats).to(DEV), torch.from_numpy(s.Ks).to(DEV), s.width, s.height)

    def render():
        kept.clear()
        if filtering is None:
            return rasterization_2dgs(*L, *cam, sh_degree=0)[0]
        return rasterization_textured_gaussians(*L, *cam, sh_degree=0, filtering=filtering)[0]

    ref = render()
    assert kept[0].contrib_masks and bool(kept[0].aniso_records) == (filtering == "anisotropic_bilinear")
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            img = render()
        assert not kept[0].contrib_masks and not kept[0].aniso_records
        assert torch.equal(img, ref)
