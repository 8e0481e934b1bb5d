"""Record sums of Gaussians that touch more tiles than the line from which their whole warp sums
them: the general form's order, slot by slot per eighth lane and then over the eight, to the
bit; the oracle's gradients within its float32 bound; the others of the warp unchanged."""
from __future__ import annotations

import pytest
import torch

from helpers import assert_grad_bounded, settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"
W, H = 640, 480  # 1200 tiles


def _scene(big):
    """70 Gaussians, in three warps; those of `big` cover the image, the others a part of it."""
    from cfgs import scenes
    sc = scenes.scene_small(n=70, width=W, height=H, seed=4)
    sc.means3D[:, :2] *= 0.3
    sc.scales = torch.full_like(sc.scales, 0.25) * torch.linspace(0.8, 1.2, 70)[:, None]
    sc.scales[big] = 6.0
    sc.opacities = torch.full_like(sc.opacities, 0.02)
    return sc


def _backward(sc, means_only=False):
    import diff_gaussian_rasterization as dgr
    from cfgs import raster
    s = sc.to(DEV)
    colors = torch.rand(sc.n, 3, generator=torch.Generator().manual_seed(2)).to(DEV)
    args = (s.means3D, s.opacities, None, colors, s.scales, s.rotations, None) if means_only else \
        (s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)
    rs = settings_for(dgr, sc)
    state = raster.forward(rs, *args)[4]
    touched = raster.inspect_state(state, W, H)["touched"].cpu()
    gc = torch.randn(3, H, W, generator=torch.Generator().manual_seed(3)).to(DEV) * 1e-4
    return raster.backward(rs, state, *args, gc, None, None, means_only=means_only), touched, gc


@pytest.mark.parametrize("big", [[5], [5, 40, 69], list(range(0, 70, 3))])
def test_long_gaussians_match_the_oracle(big):
    from oracle.c_oracle import Oracle
    from oracle.error_bound import backward_bounds
    sc = _scene(big)
    out, touched, gc = _backward(sc)
    assert (touched[big] > 1024).all()
    ref = Oracle.from_scene(sc).forward()
    want = ref.backward(gc.cpu().numpy(), magnitudes=True)
    bound = backward_bounds(ref)
    for i, key in ((0, "means2D"), (2, "opacity"), (3, "means3D"), (5, "sh"), (6, "scales"), (7, "rotations")):
        assert_grad_bounded(key, out[i].cpu(), want[key], bound[key])


@pytest.mark.parametrize("means_only", [False, True])
def test_the_others_keep_their_sums(means_only):
    """The same Gaussians with a huge, fully transparent one among them, which adds nothing to any
    pixel."""
    base, sc = _scene([]), _scene([5])
    base.opacities[5] = sc.opacities[5] = 0.0
    want, few, _ = _backward(base, means_only)
    got, touched, _ = _backward(sc, means_only)
    assert (few <= 1024).all() and int(few.max()) > 512 and int(touched[5]) > 1024
    keep = [i for i in range(70) if i != 5]
    for a, b in zip(got, want):
        if a is not None:
            assert torch.equal(a[keep], b[keep])


@pytest.mark.parametrize("big", [[], [5], [5, 40, 69]])
def test_order_of_the_sums(big):
    """The opacity and colour gradients are sums of the records alone: formed here in numpy from
    the records the render backward left."""
    import ctypes as C

    import diff_gaussian_rasterization as dgr
    import numpy as np
    from cfgs import native, raster
    sc = _scene(big)
    s = sc.to(DEV)
    colors = torch.rand(sc.n, 3, generator=torch.Generator().manual_seed(2)).to(DEV)
    args = (s.means3D, s.opacities, None, colors, s.scales, s.rotations, None)
    rs = settings_for(dgr, sc)
    state = raster.forward(rs, *args)[4]
    gc = torch.randn(3, H, W, generator=torch.Generator().manual_seed(3)).to(DEV) * 1e-4
    out = raster.backward(rs, state, *args, gc, None, None)
    lib, keep, K = native.load(), [], state.num_rendered
    scratch = torch.zeros(lib.cfgs_backward_scratch_bytes(K), dtype=torch.uint8, device=DEV)
    native.check(lib.cfgs_render_backward(C.byref(raster.make_settings(rs, keep)), sc.n, state.geom.data_ptr(),
                                          state.image.data_ptr(), state.binning.data_ptr(), K, scratch.data_ptr(),
                                          gc.data_ptr(), None, None, raster.stream_handle(gc.device)),
                 "cfgs_render_backward")
    at = (48 * K + 255) // 256 * 256
    rec = scratch[: 48 * K].view(torch.float32).reshape(K, 12).cpu().numpy()
    written = scratch[at: at + K].cpu().numpy().astype(bool)
    v = raster.inspect_state(state, W, H)
    touched, offset = v["touched"].cpu().numpy(), v["offset"].cpu().numpy()
    for g in range(sc.n):
        r = np.where(written[offset[g]: offset[g] + touched[g], None], rec[offset[g]: offset[g] + touched[g], 5:9], 0)
        lanes = np.zeros((8, 4), np.float32)
        for i in range(0, len(r), 8):
            lanes[: len(r[i:i + 8])] += r[i:i + 8].astype(np.float32)
        a = lanes[:4] + lanes[4:]
        b = a[:2] + a[2:]
        want = b[0] + b[1]
        got = np.concatenate([out[2][g].cpu().numpy(), out[1][g].cpu().numpy()])
        np.testing.assert_array_equal(got, want, err_msg=str((g, touched[g])))
