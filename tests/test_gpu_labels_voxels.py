"""The label sampler's voxel lookups where they can go wrong: samples across
brick faces, edges and corners, bricks inactive at random, outside the grid,
grids far from the origin (the 64-bit coordinates), backgrounds that are not
finite.  Labels and samples equal the oracle's bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("background", [0.75, -0.0, float("inf"), float("nan")])
@pytest.mark.parametrize("origin", [(0, 0, 0), (-13, 5, -40), (-2147483640, 7, 2147483000)])
@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 2, 5)])
def test_voxels(built, origin, dims, background):
    import gpupr_capi

    rng = np.random.default_rng(abs(hash((origin, dims))) % 2**32)
    n = int(np.prod(dims))
    table = np.where(rng.random(n) < 0.6, np.arange(n), -1).astype(np.int32)
    grid = dict(voxel_size=0.5, origin=np.array(origin, np.int32), dims=np.array(dims, np.int32),
                background=np.float32(background), table=table.reshape(dims),
                values=rng.random((n, 8, 8, 8)).astype(np.float32))
    # centroids in and around the grid, some exactly on voxels
    lo = np.array(origin, np.float64)
    c = lo + rng.uniform(-3.0, 3.0 + 8.0 * np.array(dims), (4000, 3))
    c[::3] = np.floor(c[::3])
    V = np.repeat(c * 0.5, 4, axis=0)
    T = np.arange(len(V), dtype=np.int32).reshape(-1, 4)
    want, ws = orc.sample_tet_labels(grid, V, T, (0, 0, 0), (1, 1, 1), 0.0, 0.5)
    lab, s = gpupr_capi.sample_tet_labels(grid, V, T, (0, 0, 0), (1, 1, 1), 0.0, 0.5)
    assert np.array_equal(lab, want)
    assert np.array_equal(np.isnan(s), np.isnan(ws))
    ok = ~np.isnan(ws)
    assert np.array_equal(s[ok].view(np.uint32), ws[ok].view(np.uint32))


def test_far_and_nan_vertices(built):
    import gpupr_capi

    grid = dict(voxel_size=1.0, origin=np.zeros(3, np.int32), dims=np.ones(3, np.int32),
                background=np.float32(3.0), table=np.zeros((1, 1, 1), np.int32),
                values=np.arange(512, dtype=np.float32).reshape(1, 8, 8, 8))
    V = np.array([[1e300, 2, 2], [-1e300, 2, 2], [3e9, 2, 2], [-3e9, 2, 2], [2, np.nan, 2], [2, 2, np.inf],
                  [2.5, 2.5, 2.5]], np.float64)
    T = np.repeat(np.arange(len(V), dtype=np.int32)[:, None], 4, axis=1)
    want, ws = orc.sample_tet_labels(grid, V, T, (0, 0, 0), (1, 1, 1), 0.0, 5.0)
    lab, s = gpupr_capi.sample_tet_labels(grid, V, T, (0, 0, 0), (1, 1, 1), 0.0, 5.0)
    assert np.array_equal(lab, want)
    assert np.array_equal(s, ws, equal_nan=True)
