"""The forward compositing's default launch shapes and its form for colours that are not
finite: every default (few tiles, small Gaussians, the rest) gives the bits of each explicit
schedule, and a Gaussian of infinite or NaN colour changes only the pixels it reaches."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import bits, settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _images(sc, schedule=None, colors=None):
    import diff_gaussian_rasterization as dgr
    from cfgs import autotune, raster
    s = sc.to(DEV)
    args = (settings_for(dgr, sc), s.means3D, s.opacities, None if colors is not None else s.shs, colors, s.scales,
            s.rotations, None)
    if schedule is None:
        out = raster.forward(*args)
    else:
        with autotune.using(schedule):
            out = raster.forward(*args)
    v = raster.inspect_state(out[4], sc.camera.width, sc.camera.height)
    return [out[0], out[2], out[3], v["final_T"].clone(), v["n_contrib"].clone()], out[4]


@pytest.mark.parametrize("case", ["few_tiles", "at_304_tiles", "small_gaussians", "large_gaussians"])
def test_default_shapes_are_bit_identical(case):
    from cfgs import autotune, scenes
    if case == "small_gaussians":
        sc = scenes.scene_pose(width=500, height=301, seed=4)
        sc.target = torch.zeros(3, 301, 500)
    else:
        w, h = {"few_tiles": (100, 75), "at_304_tiles": (19 * 16, 16 * 16), "large_gaussians": (500, 301)}[case]
        sc = scenes.scene_small(n=3000, width=w, height=h, seed=5)
        sc.scales = sc.scales * (5.0 if case == "large_gaussians" else 1.0)
    got, state = _images(sc)
    if case.endswith("gaussians"):  # 608 tiles: the instances per Gaussian decide
        assert (state.num_rendered < 4 * sc.n) == (case == "small_gaussians")
    for fb, fw in ((128, 4), (256, 8), (64, 4), (128, 8)):
        want, _ = _images(sc, autotune.Schedule(fb, fw, 64))
        for a, b in zip(got, want):
            assert torch.equal(a, b), (fb, fw)


@pytest.mark.parametrize("schedule", [(128, 4), (256, 8)])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_non_finite_colours_stay_where_they_are(schedule, value):
    from cfgs import autotune, scenes
    sc = scenes.scene_small(n=400, width=96, height=80, seed=6)
    g = torch.Generator().manual_seed(1)
    colors = torch.rand(400, 3, generator=g).to(DEV)
    sched = autotune.Schedule(*schedule, 64)
    base, _ = _images(sc, sched, colors)
    bad = colors.clone()
    bad[17, 1] = value
    got, _ = _images(sc, sched, bad)
    # the pixels Gaussian 17 contributes to: those whose image changes with a finite colour
    probe = colors.clone()
    probe[17, 1] += 100.0
    reached = (_images(sc, sched, probe)[0][0][1] != base[0][1])
    assert 0 < int(reached.sum()) < reached.numel()
    assert torch.equal(got[0][1][~reached], base[0][1][~reached])
    assert not bool(torch.isfinite(got[0][1][reached]).any())
    for k in (0, 2):
        np.testing.assert_array_equal(bits(got[0][k].cpu()), bits(base[0][k].cpu()))
    for a, b in zip(got[1:], base[1:]):
        assert torch.equal(a, b)
