"""The render backward where its groups can go wrong: instance counts around the eight slots
a warp sums at a time and the staging batch, ragged images, and tile counts on both sides
of the lines that pick its register budget, with and without depth and alpha gradients.
Gradients against the oracle within its float32 rounding bound (oracle.error_bound)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import assert_grad_bounded, l1_image_grad, settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"
KEYS = (("means2D", "means2D"), ("opacities", "opacity"), ("means3D", "means3D"), ("shs", "sh"), ("scales", "scales"),
        ("rotations", "rotations"))


def _check(sc, extra):
    import diff_gaussian_rasterization as dgr
    from oracle.c_oracle import Oracle
    from oracle.error_bound import backward_bounds
    s = sc.to(DEV)
    leaves = {k: getattr(s, k).clone().requires_grad_(True) for k in ("means3D", "opacities", "shs", "scales", "rotations")}
    leaves["means2D"] = torch.zeros_like(s.means3D, requires_grad=True)
    color, radii, depth, alpha = dgr.GaussianRasterizer(settings_for(dgr, sc))(**leaves)
    gc = l1_image_grad(color, s.target)
    g = torch.Generator().manual_seed(1)
    gd, ga = (torch.randn(depth.shape, generator=g).to(DEV) * 1e-3 for _ in range(2))
    if extra:
        torch.autograd.backward([color, depth, alpha], [gc, gd, ga])
    else:
        color.backward(gc)
        gd, ga = torch.zeros_like(gd), torch.zeros_like(ga)
    ref = Oracle.from_scene(sc).forward()
    want = ref.backward(gc.cpu().numpy(), gd.cpu().numpy(), ga.cpu().numpy(), magnitudes=True)
    bound = backward_bounds(ref)
    assert ref.K > 0
    for leaf, key in KEYS:
        assert_grad_bounded(leaf, leaves[leaf].grad.cpu(), want[key], bound[key])


@pytest.mark.parametrize("extra", [False, True])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 63, 64, 65, 130])
def test_slot_and_batch_edges(n, extra):
    """n large faint Gaussians over every tile of a ragged image: each warp's list has n."""
    from cfgs import scenes
    sc = scenes.scene_small(n=n, width=43, height=21, seed=n)
    sc.scales = torch.full_like(sc.scales, 0.5) * torch.linspace(0.6, 1.4, n)[:, None]
    sc.means3D[:, :2] *= 0.2
    sc.opacities = torch.full_like(sc.opacities, 0.03)
    _check(sc, extra)


@pytest.mark.parametrize("extra", [False, True])
@pytest.mark.parametrize("width,height", [(30 * 16 + 5, 20 * 16 - 3), (640, 16 * 16), (1003, 601)])
def test_register_budgets(width, height, extra):
    """620, 640 and 2394 tiles, and (below) 24: both sides of the 608-tile line."""
    from cfgs import scenes
    _check(scenes.scene_small(n=4000, width=width, height=height, seed=3), extra)
    if (width, height) == (1003, 601):
        _check(scenes.scene_small(n=4000, width=90, height=57, seed=3), extra)


@pytest.mark.parametrize("sizes", [[(320, 180)], [(640, 360), (320, 176), (90, 70)]])
def test_moments_alone_equal_the_single_path(sizes):
    """The pose batches' form (no colour sums), on both sides of its 1216-tile line, moves the
    poses exactly as the full form does in the single-solve path."""
    from cfgs import batch, pose, scenes
    probs = [pose.make_problem(scenes.scene_pose(width=w, height=h, n=4000, seed=i), DEV) for i, (w, h) in enumerate(sizes)]
    res = batch.BatchSolver(probs, use_graph=False).solve(6)
    for p, xi in zip(probs, res.xi):
        want, _ = pose.solve(p, iters=6, mode="fused")
        np.testing.assert_array_equal(xi.astype(np.float32), want.astype(np.float32))
