"""Gaussians whose instances begin exactly on the edges of the wide chunks (eight elements per
thread, 2048 positions) of a long list."""
from __future__ import annotations

import re

import pytest

import test_binning_edges_gpu as edges

pytestmark = pytest.mark.gpu


def test_starts_on_wide_chunk_edges(monkeypatch):
    from cfgs import build, raster
    text = (build.SRC_DIR / "binning.cu").read_text()
    threads = int(re.search(r"kSortThreads = (\d+);", text)[1])
    factors = re.search(r"kWideListMin = ([\d* ]+)\* kSortThreads;", text)[1]
    line = threads
    for f in factors.split("*"):
        line *= int(f)
    seen = []
    forward = raster.forward

    def counted(*a, **k):
        out = forward(*a, **k)
        seen.append(out[4].num_rendered)
        return out

    monkeypatch.setattr(raster, "forward", counted)
    monkeypatch.setitem(edges.CASES, "starts_on_chunk_edges_wide", (512, 512, 2944, 1000.0))
    edges.test_instances_equal_a_stable_sort("starts_on_chunk_edges_wide")
    # 1024 instances each, so that every second Gaussian begins on a chunk edge
    assert seen == [1024 * (2944 - len(range(5, 2944, 7)))] and seen[0] >= line
