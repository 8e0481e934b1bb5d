"""The pose kernels at the edges of their grids (1024 positions a block in the apply, 256 per
block and at most 304 summing blocks in the gradient) against float64 autograd of the
PyTorch SE(3) restatement. Tolerances: positions are three products and three additions in
float32 (6 roundings of values up to 16: 16 * 6 * 2^-24 < 6e-6); the gradient is a float64
sum rounded once (6e-8 relative, 1e-6 allowed)."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [1, 255, 257, 1023, 1025, 304 * 256, 304 * 256 + 1, 3 * 304 * 256 + 77])
def test_pose_kernels_at_grid_edges(n):
    from cfgs import pose
    g = torch.Generator().manual_seed(n)
    xi = (torch.randn(6, generator=g, dtype=torch.float64) * 0.2).float()
    xyz = (torch.randn(n, 3, generator=g) + torch.tensor([0.0, 0.0, 5.0])).clamp(-8, 8)
    gm, A = torch.randn(n, 3, generator=g), torch.randn(n, 3, 3, generator=g) * 0.3
    S = A @ A.transpose(1, 2)
    cov = torch.stack([S[:, 0, 0], S[:, 0, 1], S[:, 0, 2], S[:, 1, 1], S[:, 1, 2], S[:, 2, 2]], 1)
    gc = torch.randn(n, 6, generator=g)
    for with_cov in (False, True):
        ref = xi.double().clone().requires_grad_(True)
        m_ref, c_ref = pose.apply_pose_torch(ref, xyz.double(), cov.double() if with_cov else None)
        loss = (m_ref * gm).sum() + ((c_ref * gc).sum() if with_cov else 0.0)
        loss.backward()
        x = xi.to(DEV).requires_grad_(True)
        if with_cov:
            m, c = pose.pose_apply(x, xyz.to(DEV), cov.to(DEV))
            torch.autograd.backward([m, c], [gm.to(DEV), gc.to(DEV)])
        else:
            m = pose.pose_apply(x, xyz.to(DEV))
            m.backward(gm.to(DEV))
        assert (m.detach().cpu().double() - m_ref.detach()).abs().max() <= 6e-6
        # the covariance term's products are formed in float32 (3 x 3 products per Gaussian):
        # up to 8 roundings each of terms bounded by the sum of magnitudes
        slack = 8 * 2.0 ** -24 * 4 * float((S.abs().sum((1, 2)) * gc.abs().sum(1)).double().sum()) if with_cov else 0.0
        err = (x.grad.cpu().double() - ref.grad).abs().max()
        assert err <= 1e-6 * ref.grad.abs().max() + slack, (err, slack)
