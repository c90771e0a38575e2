"""Kernels launched with a programmatic dependency (DG_CHAIN, dg_common.cuh): frames and
sorts enqueued back to back, with nothing between them that waits, give the bits of the
same work done alone, at sizes with one CTA per kernel and with several waves of them."""

from __future__ import annotations

import numpy as np
import pytest

from diorama_gb300 import GaussianRenderer, RadixSort, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,size", [(50, (64, 48)), (20_000, (320, 240)), (300_000, (640, 360))])
def test_frames_back_to_back(device, count, size):
    raw, sh = scenes.random_gaussians(count, seed=3, half_extent=1.5)
    act = scenes.activate64(raw).astype(np.float32)
    cameras = [scenes.sphere_camera(k, *size) for k in (0, 2)]
    r = GaussianRenderer(device)
    r.setGaussians(act.reshape(-1), {"rest": sh.reshape(-1), "degree": 1})
    alone = []
    for camera in cameras:
        for _ in range(2):  # the first frame may grow the pair buffers
            r.encode(None, None, camera, (0.1, 0.2, 0.3))
            r.afterSubmit()
        alone.append(r.pixelBuffer.read(np.uint32).copy())
    for last in (0, 1):
        for k in range(40):
            r.encode(None, None, cameras[(last + k + 1) % 2], (0.1, 0.2, 0.3))
        assert np.array_equal(r.pixelBuffer.read(np.uint32), alone[last])
    assert device.check() == 0
    r.destroy()


@pytest.mark.parametrize("count", [100, 65_536, 300_000])
def test_sorts_back_to_back(device, count):
    keys = np.random.default_rng(count).integers(0, 2**32, count, dtype=np.uint64).astype(np.uint32)
    sort = RadixSort(device, count)
    sort.keys.write(keys)
    sort.values.write(np.arange(count, dtype=np.uint32))
    for _ in range(20):  # the first sorts, the others find everything in place
        sort.encode()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(sort.values.read(np.uint32), order)
    assert np.array_equal(sort.keys.read(np.uint32), keys[order])
    sort.destroy()
