"""The loss gradient's strips of 2, 4 and 6 rows (strip_rows, dg_loss.cu): bit for bit the
oracle's on both sides of the image sizes where one gives way to the next."""

from __future__ import annotations

import pytest

import test_gpu_loss_strips

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(96, 97), (96, 202), (96, 203), (96, 404), (96, 405), (200, 150), (33, 608), (33, 609)])
def test_matches_oracle(device, size):
    test_gpu_loss_strips.test_matches_oracle(device, size)
