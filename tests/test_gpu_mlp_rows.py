"""The inference kernel's loop over 128s of candidates: every candidate's score is
the same bits wherever it stands, at counts on both sides of a 128 and of the rows
that the resident CTAs take at once, and from features that are not 16-byte
aligned (the scores' values themselves: test_gpu_mlp.py)."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from diorama_gb300 import Buffer, DensifyMLP, _lib
from diorama_gb300.training import MLP_FEATURES

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 127, 128, 129, 152 * 6 * 128 - 1, 152 * 6 * 128 + 1, 300_007])
def test_scores_do_not_depend_on_the_row(device, count):
    rng = np.random.default_rng(3)
    features = np.tile(rng.normal(0, 1, (401, MLP_FEATURES)), (count // 401 + 1, 1))[:count].astype(np.float32)
    mlp = DensifyMLP(device, seed=5)
    few = mlp.predictHost(features[:401])
    got = mlp.predictHost(features)
    assert np.array_equal(got, np.tile(few, count // 401 + 1)[:count])
    # The same from an array that starts 4 bytes into an allocation.
    whole, out = device.createBuffer(features.nbytes + 16), device.createBuffer(4 * count)
    whole.write(features, 4)
    handle = ctypes.c_void_p()
    _lib.call("dg_buffer_wrap", device.handle, whole.device_pointer + 4, features.nbytes, ctypes.byref(handle))
    shifted = Buffer(device, handle, owned=True)
    mlp.predict(shifted, count, out)
    assert np.array_equal(out.read(np.float32), got)
    assert device.check() == 0
    for b in (shifted, whole, out, mlp):
        b.destroy()
