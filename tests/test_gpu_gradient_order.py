"""The order in which the blocks' sums of a splat's gradient meet (list_items_kernel,
dg_render_bwd.cu): the blocks of a chunk run together, so the one with the fewest entries
behind the splat adds first, also where more items wait than warps run.

One tile's blocks B, C and A blend 15, 155 and 253 entries behind splat S of its second
chunk; the other 380 tiles keep every warp busy. S's red gradient is 2^25 in B, -2^25 in C
and 1/2 in A: 1/2 when A adds last, 0 when it adds first (2^25 has steps of 4)."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import TileRasterizer

pytestmark = pytest.mark.gpu

SIZE, LENGTH, S = 320, 1024, 600
FAINT = 0.0045  # just over 1/255: 1024 of them leave a pixel running


def frame_splats() -> np.ndarray:
    s = np.zeros((2 * LENGTH, 12), np.float32)
    s[:, 11] = FAINT
    # Behind one another in every tile but those of the first column.
    wide = s[LENGTH:]
    wide[:, 0:2], wide[:, 3] = (168.0, 160.0), 151.9
    wide[:, 2] = 1.0 + np.arange(LENGTH) / LENGTH
    # The first tile's list: each reaches one pixel, S the whole tile.
    own = s[:LENGTH]
    own[:, 2] = 1.0 + np.arange(LENGTH) / LENGTH
    own[:, 3], own[:, 4], own[:, 6] = 2.0, 50.0, 50.0
    own[:, 0:2] = (4.5, 2.5)  # block A: rows 0 to 3 of the left half
    own[S + 1:S + 16, 0:2] = (12.5, 2.5)  # B, beside it
    own[S + 16:S + 171, 0:2] = (4.5, 6.5)  # C, below it
    own[S, 0:2], own[S, 3] = (8.0, 8.0), 7.0
    own[S, 4:7], own[S, 11] = 0.0, 0.5
    return s


def test_the_blocks_of_a_chunk_add_together(device):
    splats = frame_splats()
    pixel_grads = np.zeros((SIZE, SIZE, 4), np.float32)
    pixel_grads[0, 15, 0] = 2.0**26  # B
    pixel_grads[4, 0, 0] = -(2.0**26)  # C
    pixel_grads[0, 0, 0] = 1.0  # A
    cam = np.zeros(36, np.float32)
    cam[32:34] = SIZE
    camera, buffer, upstream = device.upload(cam), device.upload(splats), device.upload(pixel_grads)
    out = device.upload(np.zeros(splats.shape[0] * 9, np.float32))
    tiles = TileRasterizer(device, camera, buffer, splats.shape[0], 1 << 20)
    tiles.encode(None, None, (SIZE, SIZE), np.zeros(3, np.float32))
    tiles.afterSubmit()
    ranges = tiles.debugBuffers["ranges"].read(np.uint32)[:8].reshape(-1, 2)
    assert list(ranges[:2, 1] - ranges[:2, 0]) == [LENGTH, LENGTH]
    halves = 0
    for _ in range(20):
        tiles.encodeBackward(None, (SIZE, SIZE), upstream, out)
        halves += out.read(np.float32)[9 * S + 6] == 0.5
    assert halves > 10  # a warp may start late now and then
    assert device.check() == 0
    tiles.destroy()
    for b in (camera, buffer, upstream, out):
        b.destroy()
