"""The neighbour search's curve on clouds of any scale (bounds_kernel, octree_kernel,
dg_init.cu): a cloud times a power of two has the same curve, so the search takes the same
time, also where the squares of the coordinates exceed float32."""

from __future__ import annotations

import time

import numpy as np
import pytest

from diorama_gb300 import _lib

pytestmark = pytest.mark.gpu


def search(device, points):
    n = points.shape[0]
    padded = np.zeros((n, 4), np.float32)
    padded[:, :3] = points
    a, out = device.upload(padded), device.upload(np.zeros(n, np.float32))
    times = []
    for _ in range(6):
        device.synchronize()
        start = time.perf_counter()
        _lib.call("dg_mean_neighbor_distance2_buffers", device.handle, a.handle, n, out.handle)
        device.synchronize()
        times.append(time.perf_counter() - start)
    got = out.read(np.float32).copy()
    a.destroy()
    out.destroy()
    return got, min(times)


@pytest.mark.parametrize("exponent", [-40, 40, 62])
def test_a_scaled_cloud_takes_as_long(device, exponent):
    rng = np.random.default_rng(1)
    points = rng.normal(size=(100_000, 3)).astype(np.float32)
    points[17] = 1e7  # a far outlier: the curve's span is trimmed to mean +- 3 deviations
    scale = np.float32(2.0**exponent)
    got, seconds = search(device, points)
    scaled, scaled_seconds = search(device, points * scale)
    near = np.arange(points.shape[0]) != 17  # the outlier's own distances overflow
    assert np.array_equal(scaled[near], got[near] * scale * scale)
    assert scaled_seconds < 3 * seconds
    assert device.check() == 0
