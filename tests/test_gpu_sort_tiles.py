"""RadixSort's passes with tiles of 2816 keys (up to 800,000 keys) and of 3840
(dg_sort.cu), around the edges of the tiles and of the rule: a stable sort's keys and
values, for u32 and u64 keys."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import RadixSort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [70_399, 70_400, 70_401, 201_000, 800_000, 800_001])
@pytest.mark.parametrize("high_bits", [0, 16])
def test_sort(device, size, high_bits):
    rng = np.random.default_rng(size)
    keys = rng.integers(0, 2 ** (32 + high_bits), size, dtype=np.uint64)
    keys[::5] &= np.uint64(0xFF)  # many equal digits
    if not high_bits:
        keys = keys.astype(np.uint32)
    sort = RadixSort(device, size, highBits=high_bits) if high_bits else RadixSort(device, size)
    sort.keys.write(keys)
    sort.values.write(np.arange(size, dtype=np.uint32))
    sort.encode()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(sort.values.read(np.uint32), order)
    assert np.array_equal(sort.keys.read(keys.dtype), keys[order])
    assert device.check() == 0
    sort.destroy()
