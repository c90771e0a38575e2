"""The tile lists at the edge of the largest chunks (2048 splats, from 262,145 on: a second
word of hits per lane, dg_bin.cu), whole and past the capacity: as in test_gpu_bin.py."""

from __future__ import annotations

import pytest

import test_gpu_bin

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,size", [(262_144, (640, 480)), (262_145, (513, 500)), (600_000, (300, 200))])
def test_tile_lists(device, count, size):
    test_gpu_bin.test_tile_lists(device, count, size)


@pytest.mark.parametrize("share", [0.001, 0.6, 0.999])
def test_pairs_past_the_capacity(device, share):
    test_gpu_bin.test_pairs_past_the_capacity_are_dropped_in_depth_order(device, 300_001, share)
