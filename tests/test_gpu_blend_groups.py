"""The forward blend's groups of 4 staged entries (PixelBlend, dg_render.cu): images
and last indices bit for bit the oracle's loop over every entry, on lists around the
group and window sizes, with pixels that stop inside a group, opacities on both sides
of 1/255 and 0.99, means on pixel centers (a power of 0), and conics that are sharp,
flat, zero along an axis or open upwards."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from diorama_gb300 import TileRasterizer

pytestmark = pytest.mark.gpu

W, H = 40, 24


def make_splats(count: int, kind: str) -> np.ndarray:
    rng = np.random.default_rng(count * 7 + len(kind))
    s = np.zeros((count, 12), np.float32)
    s[:, 0] = rng.uniform(-4, W + 4, count)
    s[:, 1] = rng.uniform(-4, H + 4, count)
    s[::3, :2] = np.floor(s[::3, :2]) + 0.5  # on pixel centers
    s[:, 2] = rng.uniform(0.5, 2, count)  # depth
    s[:, 3] = 40.0  # radius: listed by every tile near it
    a, c = 10.0 ** rng.uniform(-3, 1, (2, count))
    b = rng.uniform(-0.95, 0.95, count) * np.sqrt(a * c)
    s[:, 8:11] = rng.uniform(0, 1, (count, 3))
    s[:, 11] = rng.choice([0.0, 1 / 255, 0.0040, 0.02, 0.3, 0.8, 0.99, 1.0, 1.5], count)
    if kind == "opaque":
        s[:, 11] = rng.uniform(0.6, 1.0, count)
        a, b, c = a * 0.01, b * 0.01, c * 0.01
    if kind == "odd":
        shape = rng.integers(0, 6, count)
        a = np.where(shape == 0, 0.0, np.where(shape == 1, -a, a))
        c = np.where(shape == 2, 0.0, np.where(shape == 3, -c, c))
        b = np.where(shape == 4, b * 3, np.where(shape == 5, -0.0, b))
    s[:, 4], s[:, 5], s[:, 6] = a, b, c
    return s


@pytest.mark.parametrize("kind", ["even", "opaque", "odd"])
@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 31, 32, 33, 36, 63, 64, 67, 130, 700])
def test_images(device, count, kind):
    splats = make_splats(count, kind)
    cam = np.zeros(36, np.float32)
    cam[32:34] = W, H
    bg = np.float32([0.2, 0.1, 0.05])
    camera, buffer = device.upload(cam), device.upload(splats)
    tiles = TileRasterizer(device, camera, buffer, count)
    for _ in range(2):  # the first frame may grow the pair buffers
        tiles.encode(None, None, (W, H), bg)
        tiles.afterSubmit()
    _, _, _, values, ranges = oracle.tile_stage(cam, splats)
    color, last, _ = oracle.rasterize(cam, bg, splats, values, ranges)
    assert np.array_equal(tiles.pixelLast.read(np.uint32)[: W * H], last)
    assert np.array_equal(tiles.pixelColor.read(np.float32)[: 4 * W * H].view(np.uint32), color.view(np.uint32))
    assert device.check() == 0
    tiles.destroy()
    camera.destroy()
    buffer.destroy()
