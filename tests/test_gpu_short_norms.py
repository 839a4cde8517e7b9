"""RMS norm of rows of one 16-byte group a thread: the last row width on either side, fewer threads than a warp, several warps."""
import pytest
import torch

from tests import test_gpu_panels as panels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [4, 124, 128, 132, 512, 996, 1024, 1028])
@pytest.mark.parametrize("m", [1, 300])
@pytest.mark.parametrize("delta", [False, True])
def test_rms_norm(gpu_ctx, h, m, delta):
    panels.test_rms_norm(gpu_ctx, h, m, delta)
