"""exp(xi) and its Jacobian blocks, formed by the lanes of one warp, around the angles where
the series take over (1e-4, 1e-3), at zero and beyond a turn, against float64 autograd of the
PyTorch restatement. Tolerances as for the kernels' grid edges: positions 6 float32 roundings
of values up to 16 (6e-6); the gradient, a float64 sum rounded once, 1e-6 relative."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("theta", [0.0, 0.9e-4, 1.1e-4, 0.9e-3, 1.1e-3, 0.5, 3.0, 20.0])
def test_pose_at_angle(theta):
    from cfgs import pose
    g = torch.Generator().manual_seed(3)
    axis = torch.tensor([0.6, -0.48, 0.64], dtype=torch.float64)
    xi = torch.cat([torch.tensor([0.3, -0.2, 0.1], dtype=torch.float64), axis * theta]).float()
    xyz = (torch.randn(700, 3, generator=g) + torch.tensor([0.0, 0.0, 5.0])).clamp(-8, 8)
    gm = torch.randn(700, 3, generator=g)
    ref = xi.double().clone().requires_grad_(True)
    m_ref = pose.apply_pose_torch(ref, xyz.double(), None)[0]
    (m_ref * gm).sum().backward()
    x = xi.to(DEV).requires_grad_(True)
    m = pose.pose_apply(x, xyz.to(DEV))
    m.backward(gm.to(DEV))
    assert (m.detach().cpu().double() - m_ref.detach()).abs().max() <= 6e-6
    assert (x.grad.cpu().double() - ref.grad).abs().max() <= 1e-6 * ref.grad.abs().max()
