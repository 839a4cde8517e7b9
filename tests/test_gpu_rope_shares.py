"""Rotary embedding and append where a token's heads are spread over several CTAs: each token on its own gives the bits of the whole portion."""
import ctypes as C

import pytest
import torch

from hf2q_b200 import decoder

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 1, 2 and more shares of a token's heads, a last share with fewer of them, portions of one CTA a token
@pytest.mark.parametrize("n_q,n_kv", [(32, 8), (8, 1), (3, 3), (64, 8)])
@pytest.mark.parametrize("m", [1, 9, 64, 100, 149, 300])
def test_portions_and_single_tokens(gpu_ctx, n_q, n_kv, m):
    S, heads = m + 7, n_q + 2 * n_kv
    src = torch.randn(m, heads * 128, generator=torch.Generator(device=DEV).manual_seed(m), device=DEV)
    outs = []
    for rows in (m, 1, 8):                                        # tokens of a call
        qkv = src.clone()
        codes, scales = [torch.zeros(n_kv, S, 128, dtype=torch.int8, device=DEV) for _ in range(2)], [torch.zeros(n_kv, S, device=DEV) for _ in range(2)]
        kv = decoder._KvCache(codes[0].data_ptr(), scales[0].data_ptr(), codes[1].data_ptr(), scales[1].data_ptr(), n_kv, 128, S)
        for at in range(0, m, rows):
            pos = torch.tensor([5 + at], dtype=torch.int32, device=DEV)
            part = qkv[at:at + rows]
            gpu_ctx._check(gpu_ctx._lib.hf2q_cuda_rope_kv_append(gpu_ctx._h, gpu_ctx._stream(), part.data_ptr(), len(part), n_q, 1e4, pos.data_ptr(), C.byref(kv)))
        outs.append([qkv, *codes, *scales])
    gpu_ctx.check_status()
    assert not torch.equal(outs[0][0], src)
    for other in outs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(outs[0], other))
