"""densify_and_prune at the edges of its blocks (1024 points a block, one gather launch over
all arrays) against the restated reference functions, and the row gather at widths around
its block size against indexing. Copies are exact; children within 1e-6 absolute, as in
test_densify_gpu.py (values of order one, a few float32 roundings of 6e-8 each)."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from test_densify_gpu import LRS, _model

pytestmark = pytest.mark.gpu
DEV = "cuda"
KW = dict(max_grad=2e-4, min_opacity=0.005, extent=3.0, max_screen_size=20, percent_dense=0.01)


def _optimizer(n, seed):
    from cfgs import densify
    p = _model(n, seed)
    g = torch.Generator().manual_seed(seed + 1)
    accum = torch.where(torch.rand(n, generator=g) < 0.5, torch.full((n,), 5e-4), torch.full((n,), 1e-5))
    opt = densify.GaussianOptimizer({k: v.to(DEV) for k, v in p.items()}, LRS)
    for k in densify.GROUPS:
        opt.exp_avg[k].copy_(torch.randn(opt.exp_avg[k].shape, generator=g))
        opt.exp_avg_sq[k].copy_(torch.rand(opt.exp_avg_sq[k].shape, generator=g))
    opt.grad_accum.copy_(accum)
    opt.denom.fill_(1.0)
    return opt, p, accum


@pytest.mark.parametrize("n", [1, 33, 1023, 1024, 1025, 2 * 1024 * 3 + 7])
def test_block_edges(n):
    from cfgs import densify
    from oracle import densify_oracle
    opt, p, accum = _optimizer(n, seed=n)
    m, v = ({k: t.cpu().clone() for k, t in d.items()} for d in (opt.exp_avg, opt.exp_avg_sq))
    splits = int(((accum >= 2e-4) & (p["scaling"].exp().max(1).values > 0.03)).sum())
    z = torch.randn(2, splits, 3, generator=torch.Generator().manual_seed(3))
    res = opt.densify_and_prune(z=z.to(DEV), **KW)
    P, M, V = densify_oracle.densify_and_prune(p, m, v, accum, torch.ones(n), z=z, **KW)
    assert res["total"] == P["xyz"].shape[0] and res["split"] == splits
    copies = res["kept"] + res["cloned"]
    for k in densify.GROUPS:
        got = opt.params[k].cpu().numpy()
        np.testing.assert_array_equal(got[:copies], P[k][:copies].numpy(), err_msg=k)
        np.testing.assert_allclose(got, P[k].numpy(), rtol=0, atol=1e-6 if k in ("xyz", "scaling") else 0, err_msg=k)
        np.testing.assert_array_equal(opt.exp_avg[k].cpu().numpy(), M[k].numpy(), err_msg=k)
        np.testing.assert_array_equal(opt.exp_avg_sq[k].cpu().numpy(), V[k].numpy(), err_msg=k)


def test_gather_widths():
    """Rows of 1 to 70,000 floats (several rows a block, one row a block, one row over the
    16-bit quotient's range), parameters and moments, in one call and one at a time."""
    from cfgs import native
    from cfgs.raster import _ptr, stream_handle
    n = 37
    opt, p, accum = _optimizer(n, seed=5)
    lib, st = native.load(), stream_handle(torch.device(DEV))
    ws = torch.empty(int(lib.cfgs_densify_workspace_bytes(n)), dtype=torch.uint8, device=DEV)
    counts = (C.c_int64 * 4)()
    native.check(lib.cfgs_densify_plan(n, _ptr(opt.grad_accum), _ptr(opt.denom), _ptr(opt.params["scaling"]),
                                       _ptr(opt.params["opacity"]), 2e-4, 0.005, 3.0, 0.01, 1, _ptr(ws), counts, st),
                 "cfgs_densify_plan")
    rows, keep = counts[0] + counts[1] + 2 * counts[3], counts[0]
    widths = [1, 2, 3, 45, 4095, 4096, 4097, 8192, 8193, 70_000]
    roles = [i % 2 for i in range(len(widths))]
    src = [torch.randn(n, w, device=DEV) for w in widths]
    idx = torch.arange(n, device=DEV, dtype=torch.float32).reshape(n, 1)  # the row map, through the same call
    arrays = [idx] + src
    out = [torch.full((rows, t.shape[1]), -1.0, device=DEV) for t in arrays]
    vp = lambda ts: (C.c_void_p * len(ts))(*[t.data_ptr() for t in ts])
    ints = lambda xs: (C.c_int32 * len(xs))(*xs)
    native.check(lib.cfgs_densify_write_many(n, _ptr(ws), counts, len(arrays), ints([1] + widths), vp(arrays), vp(out),
                                             ints([0] + roles), None, None, None, None, st), "cfgs_densify_write_many")
    rowmap = out[0].long().reshape(-1)
    assert rows > 0 and int(rowmap.min()) >= 0 and int(rowmap.max()) < n
    for s, o, w, role in zip(src, out[1:], widths, roles):
        want = s[rowmap].clone()
        if role == 1:
            want[keep:] = 0.0
        assert torch.equal(o, want), w
        single = torch.full_like(o, -1.0)
        native.check(lib.cfgs_densify_write(n, _ptr(ws), counts, w, _ptr(s), single.data_ptr(), role, None, None, None,
                                            None, st), "cfgs_densify_write")
        assert torch.equal(single, want), w
    assert lib.cfgs_densify_write(n, _ptr(ws), counts, 0, _ptr(src[0]), out[1].data_ptr(), 0, None, None, None, None,
                                  st) == 1
