"""The backward blend (rasterize_backward_kernel, dg_render_bwd.cu) on lists around its
half batches of 16 splats, batches of 32, chunks of 256 and mask windows: the splats'
gradients against the oracle's loop over every entry.

The tolerance, relative to each group's largest gradient: a pixel's transmittance is
recovered by at most 256 divisions of one ulp here (3e-5) and 700 of half an ulp in the
oracle (4e-5); the sums over pixels add less. 1e-4 covers both."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from diorama_gb300 import TileRasterizer
from test_gpu_blend_groups import H, W, make_splats

pytestmark = pytest.mark.gpu

TOLERANCE = 1e-4
GROUPS = {"mean": slice(0, 2), "conic": slice(2, 5), "opacity": slice(5, 6), "color": slice(6, 9)}


@pytest.mark.parametrize("kind", ["even", "opaque"])
@pytest.mark.parametrize("count", [1, 4, 15, 16, 17, 32, 33, 49, 255, 256, 257, 288, 513, 700])
def test_gradients(device, count, kind):
    splats = make_splats(count, kind)
    cam = np.zeros(36, np.float32)
    cam[32:34] = W, H
    bg = np.float32([0.2, 0.1, 0.05])
    pixel_grads = np.zeros((W * H, 4), np.float32)
    pixel_grads[:, :3] = np.random.default_rng(count).normal(size=(W * H, 3))
    camera, buffer, upstream = device.upload(cam), device.upload(splats), device.upload(pixel_grads)
    out = device.upload(np.zeros(count * 9, np.float32))
    tiles = TileRasterizer(device, camera, buffer, count)
    for _ in range(2):  # the first frame may grow the pair buffers
        tiles.encode(None, None, (W, H), bg)
        tiles.afterSubmit()
    for _ in range(2):  # from zero each time
        tiles.encodeBackward(None, (W, H), upstream, out)
    got = out.read(np.float32).reshape(count, 9).astype(np.float64)
    _, _, _, values, ranges = oracle.tile_stage(cam, splats)
    color, last, _ = oracle.rasterize(cam, bg, splats, values, ranges)
    frame = {"values": values, "ranges": ranges, "pixel_color": color, "pixel_last": last}
    want = oracle.rasterize_backward(cam, bg, splats.reshape(-1), frame, pixel_grads).reshape(count, 9)
    for name, columns in GROUPS.items():
        scale = np.abs(want[:, columns]).max()
        assert np.abs(got[:, columns] - want[:, columns]).max() <= TOLERANCE * scale, name
    assert device.check() == 0
    tiles.destroy()
    for b in (camera, buffer, upstream, out):
        b.destroy()
