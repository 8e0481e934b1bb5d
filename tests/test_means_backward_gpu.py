"""The backward for fixed Gaussians (only the means take gradients) against the full form: the
same bits, for every kind of colour and covariance and image gradient, on both sides of the
tile line that picks its register budget, and the full form where it does not apply."""
from __future__ import annotations

import pytest
import torch

from helpers import settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _means_grads(sc, colors, cov, used, fixed):
    import diff_gaussian_rasterization as dgr
    s = sc.to(DEV)
    leaf = lambda t: t.clone().requires_grad_(not fixed)
    m3, m2 = s.means3D.clone().requires_grad_(True), torch.zeros_like(s.means3D, requires_grad=True)
    kw = dict(colors_precomp=leaf(colors)) if colors is not None else dict(shs=leaf(s.shs))
    kw.update(dict(cov3D_precomp=leaf(cov)) if cov is not None else dict(scales=leaf(s.scales), rotations=leaf(s.rotations)))
    color, _, depth, alpha = dgr.GaussianRasterizer(settings_for(dgr, sc))(
        means3D=m3, means2D=m2, opacities=leaf(s.opacities), **kw)
    g = torch.Generator().manual_seed(4)
    outs = dict(color=color, depth=depth, alpha=alpha)
    grads = {k: torch.randn(outs[k].shape, generator=g).to(DEV) for k in ("color", "depth", "alpha")}
    torch.autograd.backward([outs[k] for k in used], [grads[k] for k in used])
    return m3.grad, m2.grad


@pytest.mark.parametrize("used", [("color",), ("color", "alpha"), ("alpha",), ("color", "depth", "alpha")])
@pytest.mark.parametrize("kind", ["sh0", "sh3", "colours", "cov"])
@pytest.mark.parametrize("width,height", [(131, 77), (1003, 601)])
def test_fixed_gaussians_give_the_same_mean_gradients(width, height, kind, used):
    from cfgs import scenes
    sc = scenes.scene_small(n=2500, width=width, height=height, seed=8, sh_degree=3 if kind == "sh3" else 0)
    g = torch.Generator().manual_seed(5)
    colors = torch.rand(2500, 3, generator=g).to(DEV) if kind in ("colours", "cov") else None
    cov = None
    if kind == "cov":
        A = torch.randn(2500, 3, 3, generator=g) * 0.05
        S = A @ A.transpose(1, 2)
        cov = torch.stack([S[:, 0, 0], S[:, 0, 1], S[:, 0, 2], S[:, 1, 1], S[:, 1, 2], S[:, 2, 2]], 1).contiguous().to(DEV)
    want = _means_grads(sc, colors, cov, used, fixed=False)
    got = _means_grads(sc, colors, cov, used, fixed=True)
    assert float(want[0].abs().sum()) > 0
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_direction_dependent_colours_are_refused():
    import diff_gaussian_rasterization as dgr
    from cfgs import raster, scenes
    sc = scenes.scene_small(n=100, width=64, height=48, seed=1, sh_degree=1)
    s = sc.to(DEV)
    args = (s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)
    rs = settings_for(dgr, sc)
    color, *_, state = raster.forward(rs, *args)
    with pytest.raises(Exception):
        raster.backward(rs, state, *args, torch.ones_like(color), None, None, means_only=True)
