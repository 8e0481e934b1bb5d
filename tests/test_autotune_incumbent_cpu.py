"""The tuner's incumbent is the schedule that a call runs under without it: a tuned call is never
slower than an untuned one by more than the noise the margin allows for. Candidates are timed
by a fake measure."""
from __future__ import annotations

import pytest


def test_the_library_says_what_its_choice_is():
    from cfgs import autotune, native
    few, small, large = (304, 16_384, 10**6), (920, 230_400, 4 * 230_400 - 1), (305, 1000, 4000)
    assert autotune.resolved(None, *few) == autotune.resolved(autotune.AUTO, *few) == autotune.Schedule(256, 8, 64)
    assert autotune.resolved(None, *small) == autotune.Schedule(256, 8, 64)
    assert autotune.resolved(None, *large) == autotune.Schedule(128, 4, 64)
    assert autotune.resolved(None, 0, 0, 0) == autotune.DEFAULT  # sizes not known
    assert autotune.resolved(autotune.Schedule(0, 0, 0, 1), *few) == autotune.Schedule(256, 8, 64, 1)
    assert autotune.resolved(autotune.Schedule(64, 4, 32), *few) == autotune.Schedule(64, 4, 32)
    lib, r, s = native.load(), native.RenderSchedule(), native.RenderSchedule()
    for bad in ((-1, 0, 0), (0, -1, 0), (0, 0, -1)):
        assert lib.cfgs_render_schedule_for(native.C.byref(s), *bad, native.C.byref(r)) == 1
    assert lib.cfgs_render_schedule_for(None, 1, 1, 1, native.C.byref(r)) == 1
    assert lib.cfgs_render_schedule_for(native.C.byref(s), 1, 1, 1, None) == 1
    with pytest.raises(RuntimeError):
        autotune.resolved(autotune.Schedule(96, 4, 64), 1, 1, 1)


@pytest.mark.parametrize("own", [(256, 8, 64), (128, 4, 64), (64, 4, 32)])
def test_nothing_faster_leaves_the_choice_to_the_library(tmp_path, own):
    from cfgs import autotune
    seen = []

    def measure(run, s):
        seen.append(s)
        return 1.0 if s == autotune.Schedule(*own) else 0.99  # faster, but inside the margin

    t = autotune.Autotuner(tmp_path / "c.json", measure=measure)
    s = t.tune("k", run=lambda: None, incumbent=autotune.Schedule(*own), unbeaten=autotune.AUTO)
    assert s == autotune.AUTO and t.lookup("k") == autotune.AUTO
    assert seen[0] == autotune.Schedule(*own) and len(set(seen)) == len(seen) == 7


def test_a_faster_shape_is_confirmed_against_the_incumbent(tmp_path):
    from cfgs import autotune
    own, best = autotune.Schedule(256, 8, 64), autotune.Schedule(128, 8, 64)
    seen = []

    def measure(run, s):
        seen.append(s)
        return 0.9 if s == best else 1.0

    t = autotune.Autotuner(tmp_path / "c.json", measure=measure)
    assert t.tune("k", run=lambda: None, incumbent=own, unbeaten=autotune.AUTO) == best
    assert seen[-4:] == [own, best, own, best]
