"""Where no shape beats the library's own choice, tuning pins none: a tuned batch or view runs
the shape it would run untuned, also where that is not the fixed default."""
from __future__ import annotations

import pytest

from helpers import settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _tuner(path):
    from cfgs import autotune
    return autotune.Autotuner(path, measure=lambda run, s: (run(), 1.0)[1])


def test_batch(tmp_path):
    from cfgs import autotune, batch, pose, scenes
    probs = [pose.make_problem(scenes.scene_pose(width=160, height=90, seed=3), DEV)]
    bs = batch.BatchSolver(probs, autotune=_tuner(tmp_path / "c.json"))
    bs.solve(2)
    assert bs.schedule_in_use() == autotune.Schedule(256, 8, 64)  # 60 tiles
    plain = batch.BatchSolver(probs)
    plain.solve(2)
    assert plain.schedule is None and plain.schedule_in_use() == bs.schedule_in_use()
    with autotune.using(autotune.Schedule(64, 4, 32)):
        assert plain.schedule_in_use() == autotune.Schedule(64, 4, 32)


def test_view(tmp_path):
    import diff_gaussian_rasterization as dgr
    from cfgs import autotune, scenes
    sc = scenes.scene_small(n=500, width=100, height=75, seed=7)
    s = sc.to(DEV)
    args = (settings_for(dgr, sc), s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)
    got = autotune.tune_rasterizer(*args, tuner=_tuner(tmp_path / "c.json"), apply=False)
    assert autotune.resolved(got, 35, 500, 10_000) == autotune.Schedule(256, 8, 64)
    assert autotune.get_schedule() == autotune.DEFAULT
