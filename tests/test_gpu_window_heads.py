"""One token of windowed attention with many heads of keys and values: clusters of every size, one CTA a head, few splits through memory."""
import pytest
import torch

from tests import test_gpu_window_decode as one

pytestmark = pytest.mark.gpu


# on 148 SMs clusters of 8, 7, 6, 5, 4, 3, 2 and 1 CTAs; the last two windows merge 3 splits and none through memory
@pytest.mark.parametrize("G,window", [(13, 2048), (14, 2048), (18, 2048), (20, 2048), (32, 2048), (43, 2048), (64, 2048), (130, 2048), (43, 9000), (150, 9000)])
@pytest.mark.parametrize("pos", [0, 300, 2047, 10000])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_one_wave(gpu_ctx, G, window, pos, dtype):
    one.test_one_token_against_64_bits(gpu_ctx, G, G, 40, 72, window, pos, dtype)
