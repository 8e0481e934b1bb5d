"""The per-Gaussian backward at the edges of its warps and blocks and of its record rounds:
Gaussian counts around 32 and 128, Gaussians of one tile to all of them in one warp (the
first 16 slots, 64 more, the rest), and one larger than many rounds. Gradients against the
oracle within its float32 rounding bound."""
from __future__ import annotations

import pytest
import torch

from test_render_bwd_edges_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [0, 3])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 128, 129, 257])
def test_warp_and_block_edges(n, degree):
    from cfgs import scenes
    sc = scenes.scene_small(n=n, width=17 * 16, height=12 * 16, seed=n, sh_degree=degree)
    sc.scales = sc.scales * torch.logspace(-1.0, 1.3, n)[torch.randperm(n, generator=torch.Generator().manual_seed(n))][:, None]
    sc.opacities = torch.full_like(sc.opacities, 0.05)
    _check(sc, True)


def test_one_large_among_small():
    from cfgs import scenes
    sc = scenes.scene_small(n=200, width=1000, height=700, seed=2)
    sc.scales[77] = 3.0
    sc.opacities = torch.full_like(sc.opacities, 0.1)
    _check(sc, False)
