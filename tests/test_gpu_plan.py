"""The blend's work plan (plan_kernel, dg_render.cu): images and last indices bit
for bit the oracle's on frames whose tiles it sends to single warps (even lists),
to whole CTAs (one list far longer than the rest) and to both, at tile counts on
both sides of the 32 tiles a CTA plans."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from diorama_gb300 import GaussianRenderer, scenes
from helpers import cam_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,size,spread", [
    (1, (1, 1), 1.0), (40, (16, 16), 1.0), (3000, (496, 16), 1.0), (3000, (512, 16), 1.0), (3000, (528, 16), 1.0),
    (6000, (130, 90), 1.0),  # a few long lists
    (20_000, (640, 360), 3.0),  # even lists
    (20_000, (640, 360), 0.02),  # nearly all splats in a few tiles
    (60_000, (320, 200), 0.6),  # opaque in front, long lists behind
])
def test_images(device, count, size, spread):
    raw, sh = scenes.random_gaussians(count, seed=11, half_extent=spread)
    act = scenes.activate64(raw).astype(np.float32)
    camera = scenes.sphere_camera(4, *size)
    r = GaussianRenderer(device)
    r.setGaussians(act.reshape(-1), {"rest": sh.reshape(-1), "degree": 1})
    for _ in range(2):  # the first frame may grow the pair buffers
        r.encode(None, None, camera, (0.2, 0.1, 0.0))
        r.afterSubmit()
    ref = oracle.render(cam_array(camera), np.float32([0.2, 0.1, 0.0]), act, sh, 1)
    pixels = size[0] * size[1]
    assert np.array_equal(r.pixelLastBuffer.read(np.uint32)[:pixels], ref["pixel_last"])
    color = r.pixelBuffer.read(np.float32)[: 4 * pixels]
    assert np.array_equal(color.view(np.uint32), ref["pixel_color"].view(np.uint32))
    assert device.check() == 0
    r.destroy()
