"""The loss gradient's strips (gradient_kernel, dg_loss.cu): gradient and pixel loss
bit for bit the oracle's where strips of 32 columns and of 6 or more rows begin and
end, and where the image is smaller than the window."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from diorama_gb300 import TrainingLoss

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [
    (1, 1), (1, 40), (40, 1), (5, 4), (31, 6), (32, 7), (33, 12), (37, 13), (64, 5), (65, 31),
    (3, 1000),  # one strip across: 912 places down
    (2000, 93),  # 63 across: 14 places down, strips of 8 rows
])
def test_matches_oracle(device, size):
    w, h = size
    rng = np.random.default_rng(w * 1000 + h)
    render = rng.uniform(-0.1, 1.2, (w * h, 4)).astype(np.float32)
    target = rng.integers(0, 256, (w * h, 4), dtype=np.uint8)
    render[w * h // 2, :3] = target[w * h // 2, :3].astype(np.float32) / np.float32(255)  # no difference
    rendered = device.upload(render)
    photo = device.createTexture(w, h)
    photo.write(target)
    loss = TrainingLoss(device, w, h)
    loss.encode(None, rendered, photo)
    _, grads, pixel_loss = oracle.loss(render, target, w, h)
    assert np.array_equal(loss.pixelGrads.read(np.float32).view(np.uint32), grads.view(np.uint32))
    assert np.array_equal(loss.pixelLoss.read(np.float32).view(np.uint32), pixel_loss.view(np.uint32))
    assert device.check() == 0
    loss.destroy()
    rendered.destroy()
    photo.destroy()
