"""debugBuffers["tileOffsets"] of a renderer's rasterizer: the tiles each splat touches,
whether the frame's tile lists are binned or sorted."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from diorama_gb300 import GaussianRenderer, scenes
from helpers import cam_array

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,size", [(1, (16, 16)), (300, (97, 61)), (5000, (640, 360)), (300, (48, 4096))])
def test_tiles_touched(device, count, size):
    raw, sh = scenes.random_gaussians(count, seed=count)
    act = scenes.activate64(raw).astype(np.float32)
    camera = scenes.sphere_camera(1, *size)
    r = GaussianRenderer(device)
    r.setGaussians(act.reshape(-1), {"rest": sh.reshape(-1), "degree": 0})
    r.encode(None, None, camera, (0, 0, 0))
    got = r.tiles.debugBuffers["tileOffsets"].read(np.uint32)[:count]
    offsets, total, *_ = oracle.tile_stage(cam_array(camera), r.splatBuffer.read(np.float32)[: count * 12])
    assert np.array_equal(got, np.diff(np.append(offsets, total)))
    r.destroy()
