"""The fused photometric loss (one pass per direction) against float64 PyTorch autograd of
the reference's loss, (1 - lambda) L1 + lambda (1 - SSIM) of the clamped image
(trainer/losses.py:98-136), at tile edges (32x32 output tiles, tensor-copy and plain
staging) and odd sizes. Tolerances: the loss is a mean of terms of order one computed in
float32 (1e-5, as the SSIM tests); the gradient 1e-4 relative with the floor of
helpers.grad_close, as the SSIM gradient tests."""
from __future__ import annotations

import pytest
import torch

from helpers import assert_grad_close

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _images(shape, seed):
    g = torch.Generator().manual_seed(seed)
    y = torch.rand(shape, generator=g)
    x = y + 0.3 * torch.randn(shape, generator=g)  # both sides of the clamp
    flat = x.reshape(-1)
    flat[:4] = torch.tensor([0.0, 1.0, -0.0, 1.5])[: flat[:4].numel()]
    flat[4:6] = y.reshape(-1)[4:6]                 # c - y = 0
    return x, y


def _reference(x, y, lam, g):
    from cfgs import pose
    xr = x.double().requires_grad_(True)
    c = xr.clamp(0, 1)
    chw = lambda t: t.reshape(-1, *t.shape[-2:])
    v = (1 - lam) * (c - y.double()).abs().mean() + lam * (1 - pose.ssim_torch(chw(c), chw(y.double())))
    (v * g).backward()
    return v.detach(), xr.grad


@pytest.mark.parametrize("shape", [(3, 32, 32), (3, 33, 36), (1, 5, 7), (3, 64, 31), (2, 3, 45, 40), (3, 97, 130)])
@pytest.mark.parametrize("lam", [0.2, 1.0])
def test_photometric_matches_float64(shape, lam):
    from cfgs import pose
    x, y = _images(shape, seed=sum(shape))
    want, dwant = _reference(x, y, lam, 0.7)
    xx = x.to(DEV).requires_grad_(True)
    v = pose.photometric_loss(xx, y.to(DEV), lam, fused=True)
    (v * 0.7).backward()
    assert abs(float(v.detach()) - float(want)) <= 1e-5
    assert_grad_close("d loss / d image", xx.grad.cpu().numpy(), dwant.numpy())
    v2 = pose.photometric_loss(x.to(DEV), y.to(DEV), lam, fused=True)
    assert float(v2) == float(v.detach())


def test_operands_outside_the_fused_form():
    """Half images, a target with a gradient and mismatched shapes take the separate calls
    and do what they did there."""
    from cfgs import pose
    from cfgs.ssim import photometric_fusable
    x, y = _images((3, 40, 44), seed=1)
    assert photometric_fusable(x.to(DEV), y.to(DEV), 0.2)
    h = x.half().to(DEV).requires_grad_(True)
    assert not photometric_fusable(h, y.to(DEV), 0.2)
    v = pose.photometric_loss(h, y.to(DEV), 0.2, fused=True)
    v.backward()
    want, _ = _reference(x.half().float(), y, 0.2, 1.0)
    assert h.grad.dtype == torch.float16 and abs(float(v.detach()) - float(want)) <= 1e-3
    with pytest.raises(NotImplementedError):
        pose.photometric_loss(x.to(DEV), y.to(DEV).requires_grad_(True), 0.2, fused=True)
    with pytest.raises(ValueError):
        pose.photometric_loss(x.to(DEV), y[:, :39].to(DEV), 0.2, fused=True)


def test_non_finite_pixels():
    """A NaN pixel makes the loss NaN and gets no gradient of its own; infinite pixels clamp."""
    from cfgs import pose
    x, y = _images((3, 40, 44), seed=2)
    x[0, 3, 4], x[1, 5, 6] = float("inf"), float("-inf")
    want, _ = _reference(x, y, 0.2, 1.0)
    xx = x.to(DEV).requires_grad_(True)
    v = pose.photometric_loss(xx, y.to(DEV), 0.2, fused=True)
    v.backward()
    assert abs(float(v.detach()) - float(want)) <= 1e-5
    assert float(xx.grad[0, 3, 4]) == 0.0 and float(xx.grad[1, 5, 6]) == 0.0 and bool(torch.isfinite(xx.grad).all())
    x[2, 7, 8] = float("nan")
    xx = x.to(DEV).requires_grad_(True)
    v = pose.photometric_loss(xx, y.to(DEV), 0.2, fused=True)
    v.backward()
    assert bool(torch.isnan(v)) and float(xx.grad[2, 7, 8]) == 0.0
