"""Training steps replayed as a graph with frames of other sizes on the trainer's renderer
between them (the graph's key, dg_train.cu): each step's image is bit for bit that of the
parameters it began with, and densification statistics count each step once."""

from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest

from diorama_gb300 import DEFAULT_SETTINGS, GaussianRenderer, RawGaussians, Trainer, TrainingView, scenes

pytestmark = pytest.mark.gpu

W, H, COUNT = 96, 64, 2000


@pytest.fixture
def trainer(device):
    raw, sh = scenes.surface_scene(COUNT, seed=3)
    cameras = [scenes.sphere_camera(k, W, H) for k in range(4)]
    rng = np.random.default_rng(1)
    images, views = [], []
    for k, camera in enumerate(cameras):
        texture = device.createTexture(W, H)
        texture.write(rng.integers(0, 256, (H, W, 4), dtype=np.uint8))
        images.append(texture)
        views.append(TrainingView(f"view {k}", camera, texture))
    t = Trainer(device, RawGaussians(raw.reshape(-1), sh.reshape(-1)), views,
                replace(DEFAULT_SETTINGS, extent=4.0, densifyUntil=0))
    t.setGraph(True)
    yield t
    t.destroy()
    for image in images:
        image.destroy()


def step_and_check(device, t):
    act, sh = t.renderer.gaussianBuffer.read(np.float32)[: COUNT * 16], t.renderer.shBuffer.read(np.float32)[: COUNT * 45]
    camera, seen = t.views[t.nextView()].camera, t.buffers["stats"].read(np.float32)[: COUNT * 4].reshape(-1, 4).copy()
    t.step()
    image = t.renderer.pixelBuffer.read(np.uint32)[: W * H * 4]
    single = GaussianRenderer(device)
    single.setGaussians(act, {"rest": sh, "degree": 0})
    for _ in range(2):  # the first frame may grow the pair buffers
        single.encode(None, None, camera, (0, 0, 0))
        single.afterSubmit()
    assert np.array_equal(image, single.pixelBuffer.read(np.uint32)[: W * H * 4])
    drawn = single.splatBuffer.read(np.float32)[: COUNT * 12].reshape(-1, 12)[:, 3] != 0
    now = t.buffers["stats"].read(np.float32)[: COUNT * 4].reshape(-1, 4)
    assert np.array_equal(now[:, 1] - seen[:, 1], drawn.astype(np.float32))
    assert not np.array_equal(t.renderer.gaussianBuffer.read(np.float32)[: COUNT * 16], act)  # it trained
    single.destroy()


@pytest.mark.parametrize("sizes", [
    [(H, W)],  # as many tiles, transposed
    [(400, 300), (W, H), (640, 480)],  # more pixels and tiles
    [(16, 700), (700, 16)],  # more bins
    [(48, 4096), (W, H)],  # a grid whose pairs are sorted
])
def test_frames_between_the_steps(device, trainer, sizes):
    step_and_check(device, trainer)
    step_and_check(device, trainer)
    for size in sizes:
        camera = scenes.sphere_camera(2, *size)
        trainer.renderer.encode(None, None, camera, (0, 0, 0))
        trainer.renderer.afterSubmit()
        step_and_check(device, trainer)
        step_and_check(device, trainer)
    assert device.check() == 0


def test_evaluations_between_the_steps(device, trainer):
    """Held-out views of one size after another, as the graph of the batch replays them."""
    rng = np.random.default_rng(2)
    for size in ((W, H), (H, W), (81, 50), (W, H)):
        image = device.createTexture(*size)
        image.write(rng.integers(0, 256, (size[1], size[0], 4), dtype=np.uint8))
        views = [TrainingView(f"held out {k}", scenes.sphere_camera(k, *size), image) for k in range(2)]
        trainer.renderer.setViewBatching(0, 0, True)
        got = trainer.evaluate(views)
        trainer.renderer.setViewBatching(0, 0, False)
        want = trainer.evaluate(views)
        assert got["psnr"] == pytest.approx(want["psnr"], rel=1e-9)  # sums in another order
        assert got["ssim"] == pytest.approx(want["ssim"], rel=1e-9)
        image.destroy()
        step_and_check(device, trainer)
    assert device.check() == 0
