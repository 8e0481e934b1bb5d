"""Frame initialisation at the edges of its blocks: kNN boxes of 32 points, super-boxes of
1024, both Morton widths; voxel runs across blocks of 1024 sorted positions. Bit-exact
against the C oracle; the sizes beyond its brute force are held to float64 distances of a
sample of queries (two float32 roundings per term of the kernel's squared distance and a
mean of three: 1e-6 relative)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from helpers import bits

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n", [31, 32, 33, 1023, 1024, 1025, 1057, 8 * 1024 + 5])
def test_knn_box_edges(n):
    from cfgs import pointcloud
    from oracle import c_oracle
    rng = np.random.default_rng(n)
    p = rng.normal(0, 1, (n, 3)).astype(np.float32)
    p[rng.integers(0, n, n // 8)] = p[0]                      # duplicates across boxes
    p[n // 2:, 2] = np.float32(0.25)                          # half of them in a plane
    got = pointcloud.dist_cuda2(torch.tensor(p, device=DEV)).cpu().numpy()
    np.testing.assert_array_equal(bits(got), bits(c_oracle.knn3_mean_dist2(p)))


def test_knn_ignores_non_finite_neighbours():
    from cfgs import pointcloud
    from oracle import c_oracle
    rng = np.random.default_rng(2)
    p = rng.normal(0, 1, (3000, 3)).astype(np.float32)
    got = pointcloud.dist_cuda2(torch.tensor(np.concatenate([p, np.full((70, 3), np.nan, np.float32)]), device=DEV))
    got = got.cpu().numpy()
    np.testing.assert_array_equal(bits(got[:3000]), bits(c_oracle.knn3_mean_dist2(p)))
    assert np.isinf(got[3000:]).all()


@pytest.mark.parametrize("n", [(1 << 18) - 3, (1 << 18) + 1, 400_003])
def test_knn_both_morton_widths(n):
    from cfgs import pointcloud
    g = torch.Generator(device=DEV).manual_seed(n)
    p = torch.randn(n, 3, device=DEV, generator=g)
    got = pointcloud.dist_cuda2(p).double()
    at = torch.randint(0, n, (300,), device=DEV, generator=g)
    d = torch.cdist(p[at].double(), p.double(), compute_mode="donot_use_mm_for_euclid_dist").square()
    d[torch.arange(300, device=DEV), at] = float("inf")
    want = torch.topk(d, 3, dim=1, largest=False).values.mean(1)
    assert bool(((got[at] - want).abs() <= 1e-6 * want).all())


@pytest.mark.parametrize("n,voxel", [(1, 0.1), (1023, 0.3), (1024, 0.3), (1025, 0.3), (5000, 50.0), (20_000, 0.013)])
def test_voxel_block_edges(n, voxel):
    """Runs inside one block, across blocks, a single voxel of every point, and single points;
    point counts of 1 to 5000 per voxel go through the reciprocal division."""
    from cfgs import pointcloud
    from oracle import c_oracle
    rng = np.random.default_rng(n)
    p = rng.uniform(-3, 3, (n, 3)).astype(np.float32)
    c = rng.uniform(0, 1, (n, 3)).astype(np.float32)
    gp, gc = pointcloud.voxel_down_sample(torch.tensor(p, device=DEV), torch.tensor(c, device=DEV), voxel)
    wp, wc = c_oracle.voxel_down_sample(p, c, voxel)
    assert gp.shape[0] == wp.shape[0]
    np.testing.assert_array_equal(bits(gp.cpu().numpy()), bits(wp))
    np.testing.assert_array_equal(bits(gc.cpu().numpy()), bits(wc))
