"""Router logits of more tiles than the chip has SMs, cut in halves and quarters, and large tiles next to the small ones that take their place."""
import pytest
import torch

from tests import test_gpu_router_tiles as tiles

pytestmark = pytest.mark.gpu


# on 148 SMs: large tiles in halves (192) and quarters (160), whole (256); small ones whole (237) and in quarters (157); fewer columns than
# the parts would need
@pytest.mark.parametrize("tokens,experts,hidden", [(8190, 384, 192), (5000, 512, 256), (8192, 512, 96), (5000, 192, 200), (9990, 60, 128), (8190, 384, 33), (8190, 384, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_logits(gpu_ctx, tokens, experts, hidden, dtype):
    tiles.test_large_tiles(gpu_ctx, tokens, experts, hidden, dtype)
