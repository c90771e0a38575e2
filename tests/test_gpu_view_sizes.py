"""One renderer's batches of views at one viewport after another (the captured graph's
key, dg_views.cu): transposed sizes with as many tiles, ragged ones, grids of other bins
and larger ones, and another scene of as many Gaussians, each bit for bit the single
frames, with the same targets and without."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import GaussianRenderer, scenes

pytestmark = pytest.mark.gpu

BACKGROUND = (0.1, 0.2, 0.3)


def scene(seed, count=3000):
    raw, sh = scenes.random_gaussians(count, seed=seed, half_extent=1.2)
    return scenes.activate64(raw).astype(np.float32), sh


def set_scene(r, seed):
    act, sh = scene(seed)
    r.setGaussians(act.reshape(-1), {"rest": sh.reshape(-1), "degree": 2})


def single_frame(r, camera):
    w, h = camera.viewport
    for _ in range(2):  # the first frame may grow the pair buffers
        r.encode(None, None, camera, BACKGROUND)
        r.afterSubmit()
    return r.pixelBuffer.read(np.uint32)[: w * h * 4]


@pytest.mark.parametrize("with_targets", [True, False])
@pytest.mark.parametrize("sizes", [
    [(490, 272), (272, 490), (481, 265), (490, 272)],  # 31 x 17 tiles, 17 x 31, 31 x 17
    [(256, 512), (128, 1024), (512, 256), (1024, 128), (256, 512)],  # 2 bins, 4, 2, 4
    [(64, 64), (16, 256), (256, 16), (250, 9), (64, 64)],  # room for all in the first guess of the pairs
    [(48, 48), (700, 500), (48, 48)],
])
def test_one_size_after_another(device, sizes, with_targets):
    r, single = GaussianRenderer(device), GaussianRenderer(device)
    pixels = max(w * h for w, h in sizes)
    targets = device.createBuffer(2 * pixels * 4) if with_targets else None
    colors = device.createBuffer(2 * pixels * 16)
    for seed in (5, 6):
        set_scene(r, seed)
        set_scene(single, seed)
        for w, h in sizes:
            cameras = [scenes.sphere_camera(k, w, h) for k in (1, 4)]
            r.renderViews(cameras, BACKGROUND, targets, colors)
            got = colors.read(np.uint32)
            for k, camera in enumerate(cameras):
                want = single_frame(single, camera)
                assert np.array_equal(got[k * want.size:(k + 1) * want.size], want), (seed, w, h, k)
    assert device.check() == 0
    r.destroy()
    single.destroy()
    for b in (targets, colors):
        if b is not None:
            b.destroy()
