"""Initial Gaussians of points or colours that autograd follows: the values of the plain call, and
the derivatives of the copies they are (positions and DC colours; zero for the other bands)."""
from __future__ import annotations

import pytest
import torch
import torch.autograd.forward_ad as fwd

pytestmark = pytest.mark.gpu
DEV = "cuda"
C0 = 0.28209479177387814


def _inputs(n=70):
    g = torch.Generator().manual_seed(n)
    return torch.randn(n, 3, generator=g).to(DEV), torch.rand(n, 3, generator=g).to(DEV)


@pytest.mark.parametrize("view_dependent", [False, True])
@pytest.mark.parametrize("degree", [0, 3])
def test_backward(degree, view_dependent):
    from cfgs import pointcloud
    p, c = _inputs()
    want = pointcloud.gaussians_from_points(p, c, degree, view_dependent)
    assert not any(t.requires_grad for t in want.values())
    pr, cr = p.clone().requires_grad_(True), c.clone().requires_grad_(True)
    got = pointcloud.gaussians_from_points(pr, cr, degree, view_dependent)
    for k, t in want.items():
        assert torch.equal(got[k], t) and got[k].shape == t.shape, k
    up = {k: torch.rand_like(t) for k, t in want.items()}
    out = [k for k in want if got[k].requires_grad]
    assert out == ["xyz", "features_dc", "features_rest"]
    gp, gc = torch.autograd.grad([got[k] for k in out], [pr, cr], [up[k] for k in out])
    assert torch.equal(gp, up["xyz"])
    assert torch.allclose(gc, up["features_dc"][:, 0] / (C0 if view_dependent else 1.0), rtol=1e-6, atol=0)
    with torch.no_grad():
        assert not any(t.requires_grad for t in pointcloud.gaussians_from_points(pr, cr, degree, view_dependent).values())


def test_forward_mode():
    from cfgs import pointcloud
    p, c = _inputs()
    tp, tc = torch.randn_like(p), torch.randn_like(c)
    with fwd.dual_level():
        got = pointcloud.gaussians_from_points(fwd.make_dual(p, tp), fwd.make_dual(c, tc), 1)
        assert torch.equal(fwd.unpack_dual(got["xyz"]).tangent, tp)
        assert torch.equal(fwd.unpack_dual(got["features_dc"]).tangent[:, 0], tc)
