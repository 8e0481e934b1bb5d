"""A pixel that an instance does not reach keeps its transmittance to the bit when the other pixel
of its pair (columns c and c + 4) is unwound: the backward divides it by 1 - 0 with the
approximate reciprocal, whose documented error of 1 ulp does not say that 1 comes out as 1."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"
W, H = 64, 48


def _gradient(pixels, depths, sigma, opacity, at):
    """Gradients of Gaussians centred on pixels, for an image gradient at one pixel alone."""
    import diff_gaussian_rasterization as dgr
    from cfgs import raster, scenes
    n = len(pixels)
    sc = scenes.scene_small(n=n, width=W, height=H, seed=0)
    z = torch.tensor(depths, dtype=torch.float32)
    xy = torch.tensor(pixels, dtype=torch.float32)
    sc.means3D = torch.stack([(xy[:, 0] + 0.5 - W / 2) * z / W, (xy[:, 1] + 0.5 - H / 2) * z / W, z], 1)
    sc.scales = (torch.tensor(sigma)[:, None] * (z / W)[:, None]).repeat(1, 3)
    sc.opacities = torch.tensor(opacity)[:, None]
    s = sc.to(DEV)
    colors = torch.linspace(0.1, 0.9, 3, device=DEV).repeat(n, 1)
    args = (s.means3D, s.opacities, None, colors, s.scales, s.rotations, None)
    rs = settings_for(dgr, sc)
    state = raster.forward(rs, *args)[4]
    seen = raster.inspect_state(state, W, H)
    assert float((seen["xy"].cpu() - xy).abs().max()) < 0.01
    gc = torch.zeros(3, H, W, device=DEV)
    gc[:, at[1], at[0]] = torch.tensor([1.0, -0.5, 0.25], device=DEV)
    out = raster.backward(rs, state, *args, gc, None, None)
    return [t[:2].cpu().numpy() for t in out if t is not None], seen["n_contrib"].reshape(H, W).cpu()


@pytest.mark.parametrize("behind", [1, 8, 200])
@pytest.mark.parametrize("x,y", [(9, 17), (13, 17), (34, 30), (38, 30)])
def test_unreached_pixel_keeps_its_transmittance(x, y, behind):
    other = x + 4 if x % 8 < 4 else x - 4
    front = [(x, y), (x, y)], [2.0, 2.5], [6.0, 6.0], [0.3, 0.6]
    want, _ = _gradient(*front, at=(x, y))
    assert all(np.isfinite(t).all() for t in want) and all((t[:, 0] != 0).all() for t in want[1:2])
    more = [(other, y)] * behind, [3.0 + 0.01 * i for i in range(behind)], [0.1] * behind, [0.05] * behind
    got, count = _gradient(*(a + b for a, b in zip(front, more)), at=(x, y))
    assert int(count[y, x]) == 2 and int(count[y, other]) > 2  # the others reach only the pair's other pixel
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)  # equal numbers (a zero's sign is the unlit pixels')
