"""The instance count's way to the host (cfgs_preprocess_counted / cfgs_wait_counts): the same
counts as cfgs_read_counts, from several threads and streams at once, after an interrupted
call, and refused for memory that is not page-locked."""
from __future__ import annotations

import ctypes as C
import threading

import pytest
import torch

from helpers import settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _forward(scene):
    import diff_gaussian_rasterization as dgr
    from cfgs import native, raster
    s = scene.to(DEV)
    out = raster.forward(settings_for(dgr, scene), s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)
    c = native.Counts()
    native.check(native.load().cfgs_read_counts(out[4].image.data_ptr(), C.byref(c),
                                                raster.stream_handle(torch.device(DEV, 0))), "cfgs_read_counts")
    return out[4].num_rendered, int(c.num_rendered)


def test_threads_and_streams():
    from cfgs import scenes
    scs = [scenes.scene_small(n=200 * (i + 1), width=64 + 16 * i, height=48, seed=i) for i in range(6)]
    want = [_forward(sc)[1] for sc in scs]
    assert len(set(want)) == len(want)
    got, errors = {}, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                got[i] = [_forward(scs[i])[0] for _ in range(40)]
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(scs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for i, k in enumerate(want):
        assert got[i] == [k] * 40


def test_interrupted_call_leaves_the_next_ones_right(monkeypatch):
    from cfgs import native, raster, scenes
    a, b = (scenes.scene_small(n=n, width=64, height=48, seed=n) for n in (300, 900))
    want = _forward(b)[1]
    lib = native.load()

    class Interrupting:
        def __getattr__(self, name):
            if name == "cfgs_depth_order":
                raise KeyboardInterrupt
            return getattr(lib, name)

    monkeypatch.setattr(native, "load", lambda: Interrupting())
    with pytest.raises(KeyboardInterrupt):
        _forward(a)
    monkeypatch.undo()
    assert _forward(b) == (want, want)
    assert _forward(a)[0] != want


def test_pageable_slot_is_refused():
    import diff_gaussian_rasterization as dgr
    from cfgs import native, raster, scenes
    sc = scenes.scene_small(n=10, width=32, height=32, seed=1)
    s, keep, lib = sc.to(DEV), [], native.load()
    cs = raster.make_settings(settings_for(dgr, sc), keep)
    g = raster.make_gaussians(s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)
    geom = torch.zeros(lib.cfgs_geom_bytes(10), dtype=torch.uint8, device=DEV)
    image = torch.zeros(lib.cfgs_image_bytes(32, 32), dtype=torch.uint8, device=DEV)
    radii = torch.zeros(10, dtype=torch.int32, device=DEV)
    ticket, st = C.c_uint32(), raster.stream_handle(torch.device(DEV, 0))
    args = (C.byref(cs), C.byref(g), geom.data_ptr(), image.data_ptr(), radii.data_ptr())
    assert lib.cfgs_preprocess_counted(*args, None, C.byref(ticket), st) == 1
    assert lib.cfgs_wait_counts(None, 1, C.byref(native.Counts()), st) == 1
    slot = torch.zeros(4, dtype=torch.int32, pin_memory=True)
    assert lib.cfgs_preprocess_counted(*args, slot.data_ptr(), C.byref(ticket), st) == 0 and ticket.value != 0
    c = native.Counts()
    assert lib.cfgs_wait_counts(slot.data_ptr(), ticket, C.byref(c), st) == 0
    # a ticket nobody will write: the wait ends with the stream, as a launch error
    assert lib.cfgs_wait_counts(slot.data_ptr(), ticket.value + 7, C.byref(c), st) == 3


@pytest.mark.parametrize("shift", [0, 4, 8, 12])
def test_counts_in_a_workspace_on_a_4_byte_boundary(shift):
    """The preprocess's 64-bit sum finds an aligned place in the image workspace's header."""
    import ctypes as C
    import diff_gaussian_rasterization as dgr
    from cfgs import native, raster, scenes
    from helpers import settings_for
    sc = scenes.scene_small(n=700, width=64, height=48, seed=3)
    s = sc.to("cuda")
    lib, keep = native.load(), []
    cs = raster.make_settings(settings_for(dgr, sc), keep)
    g = raster.make_gaussians(s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)
    geom = torch.empty(lib.cfgs_geom_bytes(700), dtype=torch.uint8, device="cuda")
    room = torch.empty(lib.cfgs_image_bytes(64, 48) + 16, dtype=torch.uint8, device="cuda")
    image, radii = room[shift:], torch.empty(700, dtype=torch.int32, device="cuda")
    stream = raster.stream_handle(s.means3D.device)
    native.check(lib.cfgs_preprocess_forward(C.byref(cs), C.byref(g), geom.data_ptr(), image.data_ptr(),
                                             radii.data_ptr(), stream), "cfgs_preprocess_forward")
    counts = native.Counts()
    native.check(lib.cfgs_read_counts(image.data_ptr(), C.byref(counts), stream), "cfgs_read_counts")
    want = raster.forward(settings_for(dgr, sc), s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)[4]
    assert counts.num_rendered == want.num_rendered > 0 and counts.flags == 0
