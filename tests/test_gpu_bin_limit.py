"""Where the pairs of a frame or of a batch pass the room for them (find_limit, dg_bin.cu):
the search for that place takes no longer than the frame's other prefix sums, also over the
rows of many views, of which every CTA searches all."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import GaussianRenderer, scenes

pytestmark = pytest.mark.gpu


def test_a_batch_past_its_capacity(device):
    w = h = 48
    views, count = 8000, 3
    raw, sh = scenes.random_gaussians(count, seed=2, half_extent=0.1)
    raw[:, 4:7] = 0.0  # each covers the frame: 9 pairs, of 4 per Gaussian that there is room for
    act = scenes.activate64(raw).astype(np.float32)
    cameras = [scenes.sphere_camera(k, w, h) for k in range(50)]
    r = GaussianRenderer(device)
    r.setGaussians(act.reshape(-1), {"rest": sh.reshape(-1), "degree": 0})
    r.setViewBatching(0, 0, False)
    colors = device.createBuffer(views * w * h * 16)
    times = []
    for _ in range(2):  # past the capacity and again in larger buffers; then once
        device.setKernelTiming(True)
        device.kernelTimingReport()
        r.renderViews([cameras[k % 50] for k in range(views)], (0, 0, 0), None, colors)
        times.append(device.kernelTimingReport()["bin_scan"])
        device.setKernelTiming(False)
    (first, both), (second, fits) = times
    assert (first, second) == (2, 1)
    assert both < 5 * fits
    got = colors.read(np.uint32).reshape(views, -1)
    for k in (0, 4000, 7999):
        for _ in range(2):
            r.encode(None, None, cameras[k % 50], (0, 0, 0))
            r.afterSubmit()
        assert np.array_equal(got[k], r.pixelBuffer.read(np.uint32)[: w * h * 4])
    r.destroy()
    colors.destroy()
