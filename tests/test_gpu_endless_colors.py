"""The backward blend with a colour that is not finite (rasterize_backward_kernel,
dg_render_bwd.cu): pixels that do not blend that splat give the gradients that they give
beside a finite colour, bit for bit, wherever the splat lies in their lists."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import TileRasterizer

pytestmark = pytest.mark.gpu

W, H = 8, 4  # one block


def gradients(device, splats):
    count = splats.shape[0]
    cam = np.zeros(36, np.float32)
    cam[32:34] = W, H
    pixel_grads = np.zeros((H, W, 4), np.float32)
    pixel_grads[:, :3, :3] = np.random.default_rng(3).normal(size=(H, 3, 3))
    camera, buffer, upstream = device.upload(cam), device.upload(splats), device.upload(pixel_grads)
    out = device.upload(np.zeros(count * 9, np.float32))
    tiles = TileRasterizer(device, camera, buffer, count)
    tiles.encode(None, None, (W, H), np.float32([0.2, 0.1, 0.05]))
    tiles.afterSubmit()
    tiles.encodeBackward(None, (W, H), upstream, out)
    got = out.read(np.float32).reshape(count, 9).copy()
    tiles.destroy()
    for b in (camera, buffer, upstream, out):
        b.destroy()
    return got


@pytest.mark.parametrize("color", [np.inf, np.nan])
@pytest.mark.parametrize("at", [0, 1, 5, 31, 32, 47, 59])
def test_only_the_pixels_that_blend_it(device, at, color):
    count = 60
    rng = np.random.default_rng(at)
    splats = np.zeros((count, 12), np.float32)
    splats[:, 0], splats[:, 1] = 1.5, 2.0  # the left half of the block
    splats[:, 2], splats[:, 3] = 1.0 + np.arange(count) / 100, 8.0
    splats[:, 4] = splats[:, 6] = 2.0
    splats[:, 8:11], splats[:, 11] = rng.uniform(0, 1, (count, 3)), 0.1
    splats[at, 0] = 7.0  # one on the right, where no gradient comes from
    other = splats.copy()
    other[at, 8:11] = color
    want, got = gradients(device, splats), gradients(device, other)
    keep = np.arange(count) != at
    assert np.isfinite(want).all() and np.abs(want[keep]).max() > 0
    assert np.array_equal(got[keep].view(np.uint32), want[keep].view(np.uint32))
    assert device.check() == 0
