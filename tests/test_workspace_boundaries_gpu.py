"""Workspaces on boundaries of their own words: a C caller may carve them out of one buffer,
at any multiple of 4 bytes (8 where they have always held 8-byte words), and gets the results
of an aligned one. The bytes around the workspace are not touched."""
from __future__ import annotations

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
GUARD = 256


def _carve(size: int, shift: int):
    """A workspace of exactly `size` bytes, `shift` bytes past a 256-byte boundary, and a check
    of the bytes before and after it."""
    room = torch.full((GUARD + size + 2 * GUARD,), 0xA5, dtype=torch.uint8, device=DEV)
    assert room.data_ptr() % 256 == 0
    ws = room[GUARD + shift: GUARD + shift + size]

    def check():
        assert bool((room[: GUARD + shift] == 0xA5).all()) and bool((room[GUARD + shift + size:] == 0xA5).all())

    return ws, check


@pytest.mark.parametrize("shift", [0, 4, 8, 12, 20])
@pytest.mark.parametrize("n", [1, 37, 1024 * 16, 1024 * 16 + 1])
def test_densify(n, shift):
    from cfgs import densify, native
    from cfgs.raster import _ptr, stream_handle
    from test_densify_edges_gpu import _optimizer
    opt, p, _ = _optimizer(n, seed=n)
    lib, st = native.load(), stream_handle(torch.device(DEV))
    ws, check = _carve(int(lib.cfgs_densify_workspace_bytes(n)), shift)
    counts = (C.c_int64 * 4)()
    native.check(lib.cfgs_densify_plan(n, _ptr(opt.grad_accum), _ptr(opt.denom), _ptr(opt.params["scaling"]),
                                       _ptr(opt.params["opacity"]), 2e-4, 0.005, 3.0, 0.01, 1, ws.data_ptr(), counts,
                                       st), "cfgs_densify_plan")
    keep, clone, split, child = (int(c) for c in counts)
    rows = keep + clone + 2 * child
    z = torch.randn(2, split, 3, generator=torch.Generator().manual_seed(1)).to(DEV)
    got = {}
    for k in ("xyz", "f_rest"):
        src = opt.params[k]
        got[k] = torch.empty((rows,) + src.shape[1:], device=DEV)
        if rows:
            native.check(lib.cfgs_densify_write(n, ws.data_ptr(), counts, src[0].numel(), _ptr(src),
                                                got[k].data_ptr(), 2 if k == "xyz" else 0, _ptr(opt.params["xyz"]),
                                                _ptr(opt.params["scaling"]), _ptr(opt.params["rotation"]), _ptr(z), st),
                         "cfgs_densify_write")
    check()
    res = opt.densify_and_prune(z=z, max_grad=2e-4, min_opacity=0.005, extent=3.0, max_screen_size=20,
                                percent_dense=0.01)
    assert (res["kept"], res["cloned"], res["split"], res["children_per_copy"]) == (keep, clone, split, child)
    for k, t in got.items():
        assert torch.equal(t, opt.params[k]), k


@pytest.mark.parametrize("shift", [0, 4, 8, 12, 24])
@pytest.mark.parametrize("shape", [(1, 5, 7), (3, 33, 36), (3, 64, 31), (3, 200, 264)])
@pytest.mark.parametrize("lam", [None, 0.2])
def test_ssim_and_photometric(shape, lam, shift):
    from cfgs import native
    from cfgs.raster import _ptr, stream_handle
    lib, st = native.load(), stream_handle(torch.device(DEV))
    g = torch.Generator().manual_seed(sum(shape))
    x, y = ((torch.rand(shape, generator=g) * 1.2 - 0.1).to(DEV) for _ in range(2))
    up = torch.full((), 0.7, device=DEV)

    def run(ws):
        out, dx = torch.empty((), device=DEV), torch.empty_like(x)
        if lam is None:
            native.check(lib.cfgs_ssim_forward(*shape, _ptr(x), _ptr(y), ws.data_ptr(), _ptr(out), st), "forward")
            native.check(lib.cfgs_ssim_backward(*shape, _ptr(x), _ptr(y), ws.data_ptr(), _ptr(up), _ptr(dx), st), "backward")
        else:
            native.check(lib.cfgs_photometric_forward(*shape, _ptr(x), _ptr(y), lam, ws.data_ptr(), _ptr(out), st),
                         "forward")
            native.check(lib.cfgs_photometric_backward(*shape, _ptr(x), _ptr(y), lam, ws.data_ptr(), _ptr(up), _ptr(dx),
                                                       st), "backward")
        return out, dx

    size = int(lib.cfgs_ssim_scratch_bytes(*shape))
    ws, check = _carve(size, shift)
    got = run(ws)
    check()
    want = run(torch.empty(size, dtype=torch.uint8, device=DEV))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
