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
