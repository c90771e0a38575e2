"""The neighbour search's tree (dg_init.cu) at the edges of its 32-point leaves and
of its levels (32, 1,024 and 32,768 points), on uniform points with far outliers,
repeated points and non-finite coordinates: bit for bit the brute force's values."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from diorama_gb300.dataset import meanNeighborDistance2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [31, 32, 33, 63, 65, 1023, 1024, 1025, 2080, 32_767, 32_769])
@pytest.mark.parametrize("odd", [False, True])
def test_leaf_and_level_edges(device, count, odd):
    rng = np.random.default_rng(count)
    points = rng.uniform(-1, 1, (count, 3)).astype(np.float32)
    if odd:
        k = max(1, count // 50)
        points[rng.integers(0, count, k)] *= np.float32(1e4)  # far outliers
        points[rng.integers(0, count, k)] = points[rng.integers(0, count, k)]  # duplicates
        points[rng.integers(0, count, 2), 0] = np.inf
        points[rng.integers(0, count, 2), 2] = -np.inf
        points[rng.integers(0, count, 2), 1] = np.nan
        points[rng.integers(0, count, 2)] = np.float32(3e30)  # distances past float32
    with np.errstate(over="ignore", invalid="ignore"):
        want = oracle.mean_neighbor_distance2(points.reshape(-1))
    assert np.array_equal(meanNeighborDistance2(device, points.reshape(-1)), want)
    assert device.check() == 0
