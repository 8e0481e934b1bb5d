"""The page-locked count slots of forwards that fail: a refused call keeps its thread's slot, an
interrupted one's is given back once its count has arrived."""
from __future__ import annotations

import pytest
import torch

from helpers import settings_for
from test_count_slot_gpu import _forward

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_refused_forwards_abandon_nothing():
    import diff_gaussian_rasterization as dgr
    from cfgs import raster, scenes
    sc = scenes.scene_small(n=200, width=64, height=48, seed=1)
    want = _forward(sc)
    s = sc.to(DEV)
    rs = settings_for(dgr, sc)._replace(sh_degree=7)
    before = len(raster._ABANDONED)
    for _ in range(20):
        with pytest.raises(RuntimeError):
            raster.forward(rs, s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)
    assert len(raster._ABANDONED) == before
    assert _forward(sc) == want


def test_interrupted_forwards_give_their_slots_back(monkeypatch):
    from cfgs import native, raster, scenes
    sc = scenes.scene_small(n=200, width=64, height=48, seed=1)
    want = _forward(sc)
    lib = native.load()

    class Interrupting:
        def __getattr__(self, name):
            if name == "cfgs_depth_order":
                raise KeyboardInterrupt
            return getattr(lib, name)

    for _ in range(20):
        monkeypatch.setattr(native, "load", lambda: Interrupting())
        with pytest.raises(KeyboardInterrupt):
            _forward(sc)
        monkeypatch.undo()
        torch.cuda.synchronize()
        assert _forward(sc) == want
    assert not raster._ABANDONED
