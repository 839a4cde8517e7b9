"""Router logits: both kernels at the edges of their tiles, parts and vector loads, against a 64-bit product."""
import pytest
import torch

import hf2q_b200 as hq
from hf2q_b200.ops import _TORCH_DT

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = hq.GpuContext(0)
    yield c
    c.close()


# up to 8 tokens: a CTA per expert; beyond: 64 x 64 tiles, columns in chunks of 32 shared by up to 8 CTAs
@pytest.mark.parametrize("tokens,experts,hidden", [(1, 1, 4), (1, 256, 2048), (3, 7, 3), (8, 5, 2052), (8, 130, 515), (9, 1, 31), (9, 64, 4096), (64, 65, 100),
                                                   (65, 32, 1024), (130, 129, 2047), (700, 256, 640), (2048, 256, 512)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shift", [0, 1])
def test_router_logits(ctx, tokens, experts, hidden, dtype, shift):
    g = torch.Generator(device="cuda").manual_seed(tokens + hidden)
    x = torch.randn(tokens * hidden + shift, generator=g, device="cuda").to(dtype)[shift:].view(tokens, hidden)      # shift: no vector loads
    w = torch.randn(experts * hidden + shift, generator=g, device="cuda")[shift:].view(experts, hidden)
    out = torch.full((tokens + 1, experts), 7.0, device="cuda")
    ctx._check(ctx._lib.hf2q_cuda_router_logits(ctx._h, ctx._stream(), x.data_ptr(), _TORCH_DT[dtype], w.data_ptr(), out.data_ptr(), tokens, experts, hidden))
    ctx.check_status()
    want, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # f32 sums of `hidden` products in any order: at most hidden roundings of 2^-24 of the sum of magnitudes each
    assert bool(((out[:tokens].double() - want).abs() <= hidden * 2.0 ** -24 * size).all())
    assert bool((out[tokens] == 7.0).all())
