"""One token of windowed attention: tiles of 16 keys, passes of 256, splits of a cluster or with a merge through memory."""
import math

import pytest
import torch

from hf2q_b200 import seqops as S
from hf2q_b200.ops import DT_BF16, DT_F32

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("H,G,d,dv", [(16, 4, 128, 128), (3, 3, 24, 40), (4, 2, 256, 256), (10, 2, 72, 136), (12, 1, 256, 200)])
@pytest.mark.parametrize("window,pos", [(2048, 0), (2048, 14), (2048, 15), (2048, 16), (2048, 255), (2048, 256), (2048, 2047), (2048, 5000), (17, 400), (256, 300),
                                        (257, 300), (3000, 2999), (9000, 700), (9000, 12000)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_one_token_against_64_bits(gpu_ctx, H, G, d, dv, window, pos, dtype):
    sop, g = S.SeqOps(gpu_ctx), torch.Generator(device=DEV).manual_seed(H * window + pos)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    cap, dp, dvp, n = window + 5, S.pad8(d), S.pad8(dv), min(pos + 1, window)
    # slots that no key of the window has hold what must not show
    kc, vc = torch.full((G, cap, dp), math.nan, dtype=dtype, device=DEV), torch.full((G, cap, dvp), math.nan, dtype=dtype, device=DEV)
    at = torch.arange(pos + 1 - n, pos, device=DEV) % cap
    k, v = torch.zeros(G, n, dp, device=DEV), torch.zeros(G, n, dvp, device=DEV)
    k[..., :d], v[..., :dv] = r(G, n, d), r(G, n, dv)
    kc[:, at], vc[:, at] = k[:, :-1].to(dtype), v[:, :-1].to(dtype)
    q, r1, r2 = r(H, d), torch.rand(H, generator=g, device=DEV), torch.rand(H, generator=g, device=DEV)
    qkv, at_pos = torch.cat([q.flatten(), k[:, -1, :d].flatten(), v[:, -1, :dv].flatten()]), torch.tensor([pos], dtype=torch.int32, device=DEV)
    a = S.struct(S.WindowAttn, qkv=qkv, ld=qkv.numel(), q_off=0, k_off=H * d, v_off=(H + G) * d, r1=r1, r2=r2, k_cache=kc, v_cache=vc, heads=H, kv_heads=G, dim=d,
                 vdim=dv, window=window, capacity=cap, cache_dtype=DT_F32 if dtype == torch.float32 else DT_BF16, scale=d ** -0.5, eps=1e-5,
                 pos=at_pos)
    out, scratch = torch.empty(1, H * dv, device=DEV), sop.window_scratch(a, DEV)
    for _ in range(2):                                            # (a second step finds the scratch as the first left it)
        sop.window_decode(a, out, scratch)
    exact = lambda t: t.to(dtype).double()
    dist = torch.arange(n - 1, -1, -1, device=DEV).double()
    rep = H // G
    s = torch.einsum("gre,gne->grn", exact(q).view(G, rep, d), exact(k[..., :d])) * d ** -0.5
    s -= (r1.double()[:, None] * torch.log1p(r2.double()[:, None] * dist)).view(G, rep, n)
    want = torch.einsum("grn,gnv->grv", torch.softmax(s, -1), exact(v[..., :dv])).reshape(1, -1)
    # f32 sums of up to 9000 products and weights: 256 eps of the values' size
    assert (out.double() - want).abs().max() < 256 * 2 ** -24 * v.abs().max()
    assert torch.equal(kc[:, pos % cap, :d], k[:, -1, :d].to(dtype)) and torch.equal(vc[:, pos % cap, :dv], v[:, -1, :dv].to(dtype))
    gpu_ctx.check_status()
