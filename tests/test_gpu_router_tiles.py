"""Router logits of many tokens: the 128 x 128 tiles, ragged in both directions, with and without vector loads."""
import pytest
import torch

from hf2q_b200.ops import _TORCH_DT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,experts,hidden", [(1300, 200, 332), (2500, 129, 96), (2433, 65, 31), (5000, 300, 64)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_large_tiles(gpu_ctx, tokens, experts, hidden, dtype):
    g = torch.Generator(device="cuda").manual_seed(tokens)
    x, w = torch.randn(tokens, hidden, generator=g, device="cuda").to(dtype), torch.randn(experts, hidden, generator=g, device="cuda")
    out = torch.full((tokens + 1, experts), 7.0, device="cuda")
    gpu_ctx._check(gpu_ctx._lib.hf2q_cuda_router_logits(gpu_ctx._h, gpu_ctx._stream(), x.data_ptr(), _TORCH_DT[dtype], w.data_ptr(), out.data_ptr(), tokens, experts, hidden))
    gpu_ctx.check_status()
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # f32 sums of `hidden` products in any order: at most hidden roundings of 2^-24 of the sum of magnitudes each
    assert bool(((out[:tokens].double() - want).abs() <= hidden * 2.0 ** -24 * size).all())
    assert bool((out[tokens] == 7.0).all())
