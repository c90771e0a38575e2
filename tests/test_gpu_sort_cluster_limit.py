"""Where the sort of u64 keys goes from one cluster to passes (CLUSTER_KEYS, dg_sort.cu):
sorted on both sides, and fewer keys do not take longer than more."""

from __future__ import annotations

import time

import numpy as np
import pytest

from diorama_gb300 import RadixSort
from test_gpu_sort_cluster import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [42_999, 43_000, 43_001])
@pytest.mark.parametrize("high_bits", [16, 32])
def test_both_sides(device, size, high_bits):
    rng = np.random.default_rng(size + high_bits)
    check(device, rng.integers(0, 2**63, size, dtype=np.uint64) >> np.uint64(31 - high_bits if high_bits < 31 else 0),
          high_bits)


@pytest.mark.parametrize("high_bits", [0, 16, 32])
def test_fewer_keys_take_no_longer(device, high_bits):
    def seconds(size):
        sort = RadixSort(device, size, highBits=high_bits)
        words = size * (2 if high_bits else 1)
        sort.keys.write(np.random.default_rng(size).integers(0, 2**32, words, dtype=np.uint64).astype(np.uint32))
        best = 1.0
        for _ in range(8):
            device.synchronize()
            start = time.perf_counter()
            for _ in range(100):
                sort.encode()
            device.synchronize()
            best = min(best, (time.perf_counter() - start) / 100)
        sort.destroy()
        return best

    times = [seconds(n) for n in (16_384, 43_000, 50_000, 65_536, 65_537)]
    assert all(few < 1.15 * max(more, 1e-5) for few, more in zip(times, times[1:])), times
