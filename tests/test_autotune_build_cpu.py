"""A tuned schedule holds for the kernels it was timed with: another build of the library does
not take it over, the same one does."""
from __future__ import annotations


def test_another_build_tunes_anew(tmp_path, monkeypatch):
    from cfgs import autotune, build
    stamp = tmp_path / "libcfgs.stamp"
    monkeypatch.setattr(build, "STAMP_PATH", stamp)
    best = {"first": autotune.Schedule(64, 4, 64), "second": autotune.Schedule(128, 8, 64)}
    calls = []

    def tuned(name):
        stamp.write_text(name + "\n")
        t = autotune.Autotuner(tmp_path / "c.json", measure=lambda run, s: (calls.append(s), 0.5 if s == best[name] else 1.0)[1])
        return t.tune("raster/n1/1x1/m1", run=lambda: None)

    assert tuned("first") == best["first"] and calls
    assert tuned("second") == best["second"]
    calls.clear()
    assert tuned("first") == best["first"] and tuned("second") == best["second"] and not calls


def test_a_library_without_a_stamp_still_tunes(tmp_path, monkeypatch):
    from cfgs import autotune, build
    monkeypatch.setattr(build, "STAMP_PATH", tmp_path / "missing")
    t = autotune.Autotuner(tmp_path / "c.json", measure=lambda run, s: 1.0)
    assert t.tune("k", run=lambda: None) == autotune.DEFAULT and t.lookup("k") == autotune.DEFAULT
