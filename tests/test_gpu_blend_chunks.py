"""The backward blend (rasterize_backward_kernel, dg_render_bwd.cu) on lists around its
chunks of 512 entries and their quarters: the splats' gradients against the oracle's loop
over every entry.

The tolerance, relative to each group's largest gradient: a pixel's transmittance is
recovered by at most 512 products with an approximate reciprocal here (an ulp and a half
each, 2^-23 x 1.5 x 512 = 9.2e-5) and by at most 1025 divisions of half an ulp in the oracle
(6.1e-5); the sums over pixels add less than 1e-5. 2e-4 covers them."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from diorama_gb300 import TileRasterizer
from test_gpu_blend_backward import GROUPS
from test_gpu_blend_groups import H, W, make_splats

pytestmark = pytest.mark.gpu

TOLERANCE = 2e-4


@pytest.mark.parametrize("kind", ["even", "faint"])
@pytest.mark.parametrize("count", [128, 129, 384, 385, 511, 512, 513, 1023, 1024, 1025])
def test_gradients(device, count, kind):
    splats = make_splats(count, kind)
    if kind == "faint":  # every pixel of every tile walks its whole list
        splats[:, 4:7] *= np.float32(1e-3)
        splats[:, 11] = np.float32(0.005)
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
    if kind == "faint":
        assert last.max() == count
    frame = {"values": values, "ranges": ranges, "pixel_color": color, "pixel_last": last}
    want = oracle.rasterize_backward(cam, bg, splats.reshape(-1), frame, pixel_grads).reshape(count, 9)
    for name, columns in GROUPS.items():
        scale = np.abs(want[:, columns]).max()
        assert np.abs(got[:, columns] - want[:, columns]).max() <= TOLERANCE * scale, name
    assert device.check() == 0
    tiles.destroy()
    for b in (camera, buffer, upstream, out):
        b.destroy()
