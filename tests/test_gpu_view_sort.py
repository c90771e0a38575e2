"""The depth sort of a batch of views (SortPlan::segments, dg_sort.cu): each view's splats
on their own, in one cluster per view or in passes over all views, at counts on both
sides of the sort's tiles and of the cluster's room. Images are those of single frames."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import GaussianRenderer, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views,count", [(1, 1), (2, 31), (3, 3841), (12, 200), (20, 5000), (2, 65_536), (2, 65_537),
                                         (9, 70_001)])
def test_images(device, views, count):
    w, h = 96, 64
    raw, sh = scenes.random_gaussians(count, seed=views, half_extent=1.5)
    raw[2::3, :3] = raw[1::3, :3][: raw[2::3].shape[0]]  # equal depths stay in index order
    act = scenes.activate64(raw).astype(np.float32)
    cameras = [scenes.sphere_camera(k, w, h) for k in range(views)]
    r = GaussianRenderer(device)
    r.setGaussians(act.reshape(-1), {"rest": sh.reshape(-1), "degree": 1})
    colors = device.upload(np.zeros((views, h, w, 4), np.float32))
    r.setViewBatching(views)
    for _ in range(2):
        r.renderViews(cameras, (0.1, 0.2, 0.3), None, colors)
    got = colors.read(np.uint32).reshape(views, -1)
    for k, camera in enumerate(cameras):
        for _ in range(2):  # the first frame may grow the pair buffers
            r.encode(None, None, camera, (0.1, 0.2, 0.3))
            r.afterSubmit()
        assert np.array_equal(got[k], r.pixelBuffer.read(np.uint32)[: w * h * 4]), k
    assert device.check() == 0
    r.destroy()
    colors.destroy()
