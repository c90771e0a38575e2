"""More views in one call than a launch takes (MAX_BATCH, dg_views.cu): the images of the
views around the limit are those of single frames."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import GaussianRenderer, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views", [65_535, 65_537])
def test_views_past_the_launch_limit(device, views):
    w = h = 16
    raw, sh = scenes.random_gaussians(3, seed=2, half_extent=0.5)
    act = scenes.activate64(raw).astype(np.float32)
    cameras = [scenes.sphere_camera(k, w, h) for k in range(61)]
    r = GaussianRenderer(device)
    r.setGaussians(act.reshape(-1), {"rest": sh.reshape(-1), "degree": 1})
    colors = device.createBuffer(views * w * h * 16)
    r.renderViews([cameras[k % 61] for k in range(views)], (0.1, 0.2, 0.3), None, colors)
    got = colors.read(np.uint32).reshape(views, -1)
    for k in (0, 1, 65_533, 65_534, views - 2, views - 1):
        r.encode(None, None, cameras[k % 61], (0.1, 0.2, 0.3))
        assert np.array_equal(got[k], r.pixelBuffer.read(np.uint32)[: w * h * 4]), k
    assert device.check() == 0
    r.destroy()
    colors.destroy()
