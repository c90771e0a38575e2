"""PrefixSum in one launch (up to 4096 values) and in two (dg_scan.cu): lengths and
device-side counts on both sides of the 4096-value tiles, scans enqueued back to back,
and sums that wrap."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import PrefixSum

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity,n", [(1, 1), (4096, 0), (4096, 4096), (8192, 4096), (8192, 4097), (8192, 8192),
                                        (8193, 0), (8193, 8193), (1_100_003, 1_099_999), (1_100_003, 5)])
@pytest.mark.parametrize("device_count", [False, True])
def test_counts(device, capacity, n, device_count):
    if not device_count:
        n = capacity
    values = np.random.default_rng(capacity + n).integers(0, 2**32, capacity, dtype=np.uint64).astype(np.uint32)
    buf = device.upload(values)
    count = device.upload(np.array([n], np.uint32)) if device_count else None
    scan = PrefixSum(device, buf, capacity, count)
    want = values.copy()
    for _ in range(3):  # each scans what the one before left
        scan.encode()
        total = int(want[:n].sum(dtype=np.uint64)) & 0xFFFFFFFF
        want[:n] = np.concatenate([np.zeros(min(n, 1), np.uint64), np.cumsum(want[:n], dtype=np.uint64)[:-1]])
    assert np.array_equal(buf.read(np.uint32), want)
    assert int(scan.total.read(np.uint32)[0]) == total
    assert device.check() == 0
    scan.destroy()
    buf.destroy()
    if count:
        count.destroy()
