"""RadixSort in one cluster (sort_cluster_kernel, dg_sort.cu) and at the sizes where
the passes take over: keys and values are those of a stable sort, on random keys, keys
with few digits (every lane of a warp counts the same one) and a device-side count."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import RadixSort

pytestmark = pytest.mark.gpu

SIZES_32 = [1, 2, 31, 32, 33, 511, 513, 8191, 8193, 65_535, 65_536, 65_537]
SIZES_64 = [1, 33, 8193, 65_536, 65_537]


def check(device, keys, high_bits, used=None):
    count = device.upload(np.array([used], np.uint32)) if used is not None else None
    sort = RadixSort(device, keys.size, highBits=high_bits, count=count) if high_bits else \
        RadixSort(device, keys.size, count=count)
    values = np.random.default_rng(1).permutation(keys.size).astype(np.uint32)
    sort.keys.write(keys)
    sort.values.write(values)
    sort.encode()
    n = keys.size if used is None else used
    order = np.argsort(keys[:n], kind="stable")
    assert np.array_equal(sort.values.read(np.uint32), np.concatenate([values[:n][order], values[n:]]))
    assert np.array_equal(sort.keys.read(keys.dtype), np.concatenate([keys[:n][order], keys[n:]]))
    assert device.check() == 0
    sort.destroy()
    if count:
        count.destroy()


@pytest.mark.parametrize("size", SIZES_32)
@pytest.mark.parametrize("few", [False, True])
def test_u32(device, size, few):
    rng = np.random.default_rng(size)
    keys = rng.integers(0, 2**32, size, dtype=np.uint64).astype(np.uint32)
    if few:
        keys = np.uint32(0x3F800000) + (keys & np.uint32(0x00010003))
    check(device, keys, 0)


@pytest.mark.parametrize("size", SIZES_64)
@pytest.mark.parametrize("high_bits", [8, 16])
def test_u64(device, size, high_bits):
    rng = np.random.default_rng(size + high_bits)
    keys = rng.integers(0, 2 ** (32 + high_bits), size, dtype=np.uint64)
    keys[::3] &= np.uint64(0xFF000000FF)
    check(device, keys, high_bits)


@pytest.mark.parametrize("used", [0, 1, 511, 60_000])
def test_device_count(device, used):
    keys = np.random.default_rng(used).integers(0, 2**32, 60_000, dtype=np.uint64).astype(np.uint32)
    check(device, keys, 0, used)
