"""The tile lists of depth-ordered splats (dg_bin.cu) at the edges of its chunks
(256 splats; 512 from 65,537 splats on), its 16 x 16-tile bins and the largest
grids it takes, and past them, where the pairs are sorted instead: total, lists,
ranges and keys bit for bit against the oracle's stable sort. With too little room
for the frame's pairs, the ones that come first in depth order are listed."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from diorama_gb300 import GaussianRenderer, scenes
from helpers import cam_array

pytestmark = pytest.mark.gpu


def scene(count: int, half_extent: float = 2.0):
    raw, sh = scenes.random_gaussians(count, seed=count % 991, half_extent=half_extent)
    raw[2::3, :3] = raw[1::3, :3][: raw[2::3].shape[0]]  # equal depths
    return scenes.activate64(raw).astype(np.float32), sh


def frame(device, act, sh, camera, capacity=None):
    r = GaussianRenderer(device, {"initialPairCapacity": capacity} if capacity else None)
    r.setGaussians(act.reshape(-1), {"rest": sh.reshape(-1), "degree": 0})
    r.encode(None, None, camera, (0, 0, 0))
    return r


@pytest.mark.parametrize("count,size", [
    (1, (16, 16)), (255, (1, 1)), (256, (256, 256)), (257, (257, 255)), (2049, (272, 16)), (3000, (16, 272)),
    (65_536, (640, 480)), (65_537, (513, 500)), (131_073, (33, 700)),
    (700, (4080, 64)), (700, (4081, 64)), (700, (48, 4080)), (700, (48, 4096)),  # 255 tiles a side, and 256
    (900, (2048, 2048)), (900, (2064, 2048)),  # 16,384 tiles, and more
])
def test_tile_lists(device, count, size):
    act, sh = scene(count)
    camera = scenes.sphere_camera(2, *size)
    r = frame(device, act, sh, camera)
    r.afterSubmit()
    r.encode(None, None, camera, (0, 0, 0))
    r.afterSubmit()
    splats = r.splatBuffer.read(np.float32)[: count * 12]
    _, total, keys, values, ranges = oracle.tile_stage(cam_array(camera), splats)
    debug = r.tiles.debugBuffers
    assert int(debug["pairTotal"].read(np.uint32)[0]) == total == r.tiles.lastPairCount
    assert np.array_equal(debug["ranges"].read(np.uint32)[: ranges.size], ranges)
    assert np.array_equal(debug["pairSplats"].read(np.uint32)[:total], values)
    assert np.array_equal(debug["pairKeys"].read(np.uint64)[:total], keys)
    assert device.check() == 0
    r.destroy()


@pytest.mark.parametrize("count,share", [(300, 0.0), (3000, 0.37), (3000, 0.999), (70_000, 0.5)])
def test_pairs_past_the_capacity_are_dropped_in_depth_order(device, count, share):
    act, sh = scene(count)
    camera = scenes.sphere_camera(3, 320, 240)
    whole = frame(device, act, sh, camera)
    whole.afterSubmit()
    splats = whole.splatBuffer.read(np.float32)[: count * 12]
    _, total, keys, values, _ = oracle.tile_stage(cam_array(camera), splats)
    whole.destroy()
    capacity = max(1, int(total * share))
    r = frame(device, act, sh, camera, capacity)
    # The pairs in the order they are dropped from: by depth, then splat, then tile.
    kept = np.lexsort((keys >> np.uint64(32), values, keys & np.uint64(0xFFFFFFFF)))[:capacity]
    kept = np.sort(kept)  # back to the sorted keys' order
    tiles = (keys[kept] >> np.uint64(32)).astype(np.int64)
    grid = 20 * 15
    starts, ends = np.searchsorted(tiles, np.arange(grid)), np.searchsorted(tiles, np.arange(grid), "right")
    ranges = np.stack([starts, ends], 1)
    ranges[starts == ends] = 0
    debug = r.tiles.debugBuffers
    assert int(debug["pairTotal"].read(np.uint32)[0]) == total > capacity
    assert np.array_equal(debug["ranges"].read(np.uint32)[: 2 * grid], ranges.reshape(-1))
    assert np.array_equal(debug["pairSplats"].read(np.uint32)[:capacity], values[kept])
    r.afterSubmit()
    assert r.tiles.pairCapacity >= total == r.tiles.lastPairCount
    assert device.check() == 0
    r.destroy()
