"""Values that are not finite: they stay with the pixels and Gaussians they belong to, and are
no error of the call."""
from __future__ import annotations

import ctypes as C

import pytest
import torch

from helpers import settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_non_finite_colours_raise_no_flag(value):
    """A caller that takes any flag for an error accepts a view with such a colour."""
    import diff_gaussian_rasterization as dgr
    from cfgs import native, raster, scenes
    sc = scenes.scene_small(n=300, width=64, height=48, seed=2)
    s = sc.to(DEV)
    colors = torch.rand(300, 3, generator=torch.Generator().manual_seed(1)).to(DEV)
    colors[::3, 1] = value
    state = raster.forward(settings_for(dgr, sc), s.means3D, s.opacities, None, colors, s.scales, s.rotations, None)[4]
    counts = native.Counts()
    native.check(native.load().cfgs_read_counts(state.image.data_ptr(), C.byref(counts),
                                                raster.stream_handle(s.means3D.device)), "cfgs_read_counts")
    assert counts.num_rendered == state.num_rendered > 0 and counts.flags == 0


def _gradients(sc, colors, gc, gd=None, ga=None, means_only=False):
    """The seven gradient arrays (the means' two) of one render with precomputed colours."""
    import diff_gaussian_rasterization as dgr
    from cfgs import raster
    s = sc.to(DEV)
    args = (s.means3D, s.opacities, None, colors, s.scales, s.rotations, None)
    rs = settings_for(dgr, sc)
    state = raster.forward(rs, *args)[4]
    out = raster.backward(rs, state, *args, gc, gd, ga, means_only=means_only)
    return {k: t for k, t in zip(("means2D", "colors", "opacity", "means3D", "cov3D", "sh", "scales", "rotations"), out)
            if t is not None}


def _scene(n=1500):
    from cfgs import scenes
    sc = scenes.scene_small(n=n, width=90, height=70, seed=8)
    g = torch.Generator().manual_seed(3)
    colors = torch.rand(n, 3, generator=g).to(DEV)
    images = [(torch.randn(c, 70, 90, generator=g) * 1e-2).to(DEV) for c in (3, 1, 1)]
    return sc, colors, images


def _reaching(sc, colors, mask):
    """Gaussians that contribute to a pixel of the mask: theirs is a colour gradient."""
    ones = mask.to(torch.float32).expand(3, -1, -1).contiguous()
    return (_gradients(sc, colors, ones)["colors"] != 0).any(1)


@pytest.mark.parametrize("pixel", [(37, 41), (33, 45), (20, 60), (50, 30)])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("form,plane", [("colour", 0), ("depth", 0), ("depth", 1), ("depth", 2), ("means", 0), ("means", 2)])
def test_a_bad_image_gradient_stays_with_its_gaussians(form, plane, value, pixel):
    """One pixel's gradient is not finite: the Gaussians that do not contribute to that pixel keep
    their gradients, those that do have no finite one left in the sums it enters."""
    sc, colors, images = _scene()
    pick = lambda im: (im[0], im[1] if form == "depth" else None, im[2] if plane == 2 or form == "depth" else None)
    want = _gradients(sc, colors, *pick(images), means_only=form == "means")
    bad = [t.clone() for t in images]
    bad[plane][(slice(0, 1),) + pixel] = value
    got = _gradients(sc, colors, *pick(bad), means_only=form == "means")
    mask = torch.zeros(1, 70, 90, dtype=torch.bool, device=DEV)
    mask[(0,) + pixel] = True
    at = _reaching(sc, colors, mask)
    assert 0 < int(at.sum()) < sc.n // 4
    for k in want:
        assert torch.isfinite(want[k]).all()
        assert torch.equal(got[k][~at], want[k][~at]), k
    assert not torch.isfinite(got["means3D"][at]).all(1).any()
    if plane == 0 and form != "means":
        assert not torch.isfinite(got["colors"][at, 0]).any()
        assert torch.equal(got["colors"][:, 1:], want["colors"][:, 1:])
    if plane > 0 and form == "depth":
        assert torch.equal(got["colors"], want["colors"])


@pytest.mark.parametrize("value", [float("nan"), float("-inf")])
@pytest.mark.parametrize("form", ["colour", "depth", "means"])
def test_a_bad_colour_stays_with_its_pixels(form, value):
    """One Gaussian's colour is not finite: those that contribute to none of its pixels keep their
    gradients."""
    sc, colors, images = _scene()
    images = (images[0], images[1] if form == "depth" else None, None)
    want = _gradients(sc, colors, *images, means_only=form == "means")
    one = torch.zeros_like(colors)
    one[17] = 1.0
    import diff_gaussian_rasterization as dgr
    from cfgs import raster
    s = sc.to(DEV)
    own = raster.forward(settings_for(dgr, sc), s.means3D, s.opacities, None, one, s.scales, s.rotations, None)[0]
    near = _reaching(sc, colors, own[:1] > 0)
    assert bool(near[17]) and int(near.sum()) < sc.n // 2
    bad = colors.clone()
    bad[17, 2] = value
    got = _gradients(sc, bad, *images, means_only=form == "means")
    for k in want:
        assert torch.equal(got[k][~near], want[k][~near]), k
