"""The binning's instance list at the sizes where its chunks can go wrong, against the same
list built and sorted with numpy from the Gaussians' rectangles and depths (whole numbers:
equal)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import settings_for

pytestmark = pytest.mark.gpu
DEV = "cuda"

# image, Gaussians, size factor, depth range: instances per Gaussian, tile passes and the
# position of Gaussian starts in a chunk follow from them
CASES = {
    "one_gaussian": (64, 48, 1, 1.0),
    "one_tile": (16, 16, 300, 1.0),
    "below_one_chunk_one_pass": (200, 150, 40, 1.0),
    "one_pass_ragged": (255, 249, 9_000, 1.0),
    "starts_on_chunk_edges": (512, 512, 7, 1000.0),          # every Gaussian: all 1024 tiles
    "starts_on_chunk_edges_long": (512, 512, 640, 1000.0),   # above the wide chunks' line
    "one_over_many_chunks": (1920, 1080, 2, 1000.0),         # 8160 tiles each
    "long_two_pass": (1000, 620, 40_000, 4.0),
    "three_pass": (4112, 4112, 3_000, 3.0),                  # 257 * 257 tiles
    "three_pass_giant": (4112, 4112, 12, 1000.0),
    "equal_depths": (320, 240, 5_000, 2.0),
    "depth_chunks_added_up": (100, 80, 128 * 1024, 0.3),     # last count without a scan launch
    "depth_chunks_scanned": (100, 80, 128 * 1024 + 1, 0.3),
}


@pytest.mark.parametrize("case", list(CASES))
def test_instances_equal_a_stable_sort(case):
    import diff_gaussian_rasterization as dgr
    from cfgs import raster, scenes
    w, h, n, factor = CASES[case]
    sc = scenes.scene_small(n=n, width=w, height=h, seed=len(case))
    sc.scales = sc.scales * factor
    if case == "equal_depths":
        sc.means3D[:, 2] = 3.0 + 0.5 * (torch.arange(n) % 3).float()
    if n > 30:
        sc.means3D[5::7, 2] = -1.0  # behind the camera: no instances
    s = sc.to(DEV)
    state = raster.forward(settings_for(dgr, sc), s.means3D, s.opacities, s.shs, None, s.scales, s.rotations, None)[4]
    v = {k: t.cpu().numpy() for k, t in raster.inspect_state(state, w, h).items()}
    touched = v["touched"].astype(np.int64)
    K, gx, tiles = int(touched.sum()), (w + 15) // 16, ((w + 15) // 16) * ((h + 15) // 16)
    assert K == state.num_rendered
    if case.startswith("starts_on_chunk_edges"):
        live = touched > 0
        assert live.all() or n > 30
        assert (touched[live] == 1024).all()

    order = np.nonzero(touched)[0]
    order = order[np.argsort(v["rgbd"][order, 3], kind="stable")]
    first = np.concatenate([[0], np.cumsum(touched[order])])
    gid = np.repeat(order, touched[order])
    j = np.arange(K) - np.repeat(first[:-1], touched[order])
    rect = v["rect"].astype(np.int64)
    x0, y0, x1 = rect[gid, 0] & 0xffff, (rect[gid, 0] >> 16) & 0xffff, rect[gid, 1] & 0xffff
    tile = (y0 + j // (x1 - x0)) * gx + x0 + j % (x1 - x0)
    by_tile = np.argsort(tile, kind="stable")
    np.testing.assert_array_equal(v["offset"][order], first[:-1])
    np.testing.assert_array_equal(v["sorted_gid"], gid[by_tile])
    np.testing.assert_array_equal(v["sorted_pidx"], by_tile)
    np.testing.assert_array_equal(v["tile_range"], np.concatenate([[0], np.cumsum(np.bincount(tile, minlength=tiles))]))
