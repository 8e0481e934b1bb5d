"""The default compositing shape goes by the Gaussians that touch a tile, whose number comes with
the instance count: culled ones are none of a view's small Gaussians."""
from __future__ import annotations

import pytest
import torch

from helpers import settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("culled", [0.0, 0.9, 1.0])
@pytest.mark.parametrize("scale,small", [(0.1, True), (1.0, False)])
def test_culled_gaussians_do_not_count(culled, scale, small, monkeypatch):
    import diff_gaussian_rasterization as dgr
    from cfgs import autotune, native, raster, scenes
    sc = scenes.scene_small(n=4000, width=640, height=480, seed=3)  # 1200 tiles
    sc.scales = sc.scales * scale
    k = int(4000 * culled)
    sc.means3D[:k, 2] = -1.0
    s = sc.to(DEV)
    lib, seen = native.load(), []

    class Spy:
        def __getattr__(self, name):
            fn = getattr(lib, name)
            if name != "cfgs_composite_forward":
                return fn

            def call(settings, *a):
                seen.append(settings._obj.schedule.fwd_warps)
                return fn(settings, *a)
            return call

    monkeypatch.setattr(native, "load", lambda: Spy())
    args = (settings_for(dgr, sc), s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)
    state = raster.forward(*args)[4]
    monkeypatch.undo()
    touching = raster.touching(state)
    assert touching == int((raster.inspect_state(state, 640, 480)["touched"] > 0).sum())
    assert (touching > 0) == (culled < 1.0)
    if culled < 1.0:
        assert (state.num_rendered < 4 * touching) == small
        assert seen == [8 if small else 4]
        assert seen == [autotune.resolved(None, 1200, touching, state.num_rendered).fwd_warps]
    with autotune.using(autotune.Schedule(64, 4, 32)):  # a chosen shape stays
        monkeypatch.setattr(native, "load", lambda: Spy())
        raster.forward(*args)
        assert seen[-1] == 4


def test_batches_count_them_too():
    from cfgs import autotune, batch, pose, scenes
    sc = scenes.scene_pose(width=640, height=360, seed=2)
    shape = {}
    for culled in (0, 1):
        p = pose.make_problem(sc, DEV)
        if culled:  # a tenth of the Gaussians is left, with ten times the size
            p.xyz = p.xyz.clone()
            p.xyz[torch.arange(p.xyz.shape[0], device=DEV) % 10 != 0, 2] = -1.0
            p.scales = p.scales * 10.0
        bs = batch.BatchSolver([p], use_graph=False)
        bs.solve(2)
        shape[culled] = bs.schedule_in_use()
        assert 0 < bs.touching <= p.xyz.shape[0]
    assert shape[0] == autotune.Schedule(256, 8, 64) and shape[1] == autotune.Schedule(128, 4, 64)
