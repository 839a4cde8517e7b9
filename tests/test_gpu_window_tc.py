"""Windowed attention over many query tiles on tcgen05: windows and portions around the tile sizes (128 queries, 64 keys)."""
import numpy as np
import pytest
import torch

from hf2q_b200 import seqops as S
from oracle import fomatar_forward as F
from tests.test_gpu_seqops import rel, run_window

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,d,dv,window,bias", [(2, 1, 72, 128, 1, True), (3, 3, 128, 100, 63, False), (4, 2, 96, 65, 128, True), (2, 2, 128, 128, 129, False),
                                                  (1, 1, 127, 9, 300, True), (8, 2, 65, 120, 2000, False)])
def test_many_tiles(gpu_ctx, H, G, d, dv, window, bias):
    rng, T = np.random.default_rng(d + window), 643
    q, k, v = 2 * rng.standard_normal((T, H, d)), rng.standard_normal((T, G, d)), rng.standard_normal((T, G, dv))
    r1, r2 = (rng.random(H) + 0.2, rng.random(H) * 0.3) if bias else (None, None)
    to = lambda x: torch.tensor(x).to(torch.bfloat16).double().numpy()
    q, k, v = to(q), to(k), to(v)
    want = F.window_attention(q, k, v, window, d ** -0.5, r1 if bias else np.zeros(H), r2 if bias else np.zeros(H)).reshape(T, -1)
    for cuts in ([T], [127, 128, 129, 2, 257], [385, 258]):
        got = run_window(S.SeqOps(gpu_ctx), q, k, v, window, d ** -0.5, r1, r2, torch.bfloat16, cuts)
        gpu_ctx.check_status()
        assert rel(got, want) < 2 ** -8, cuts            # probabilities rounded to bf16 (2^-9 each), and their sum not


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("which", ["k", "v"])
@pytest.mark.parametrize("H,d,dv,window,at", [(2, 128, 128, 500, 70), (2, 120, 121, 257, 11), (32, 72, 128, 600, 255), (32, 128, 65, 512, 127)])
def test_hidden_keys_do_not_reach_a_row(gpu_ctx, bad, which, H, d, dv, window, at):
    """A key or value that is not finite shows in the queries that see it and in no other of the tile, before it or past its window."""
    rng, T = np.random.default_rng(d + window), 300
    to = lambda x: torch.tensor(x).to(torch.bfloat16).double().numpy()
    q, k, v = (to(rng.standard_normal((T, H, n))) for n in (d, d, dv))
    r1, r2 = rng.random(H) + 0.2, rng.random(H) * 0.3
    want = F.window_attention(q, k, v, window, d ** -0.5, r1, r2).reshape(T, -1)
    {"k": k, "v": v}[which][at, :, 5] = bad
    blind = np.ones(T, bool)
    blind[at:at + window] = False
    got = run_window(S.SeqOps(gpu_ctx), q, k, v, window, d ** -0.5, r1, r2, torch.bfloat16, [T])
    gpu_ctx.check_status()
    assert rel(got[torch.tensor(blind)], want[blind]) < 2 ** -8
    if which == "v":
        assert not got[at:min(at + window, T)].view(-1, H, dv)[:, :, 5].isfinite().any()


# where the choice between the two kernels lies: by window, by tiles per SM, by the size of a key and a value
@pytest.mark.parametrize("H,G,d,dv,window,T", [(2, 1, 128, 128, 256, 400), (2, 1, 128, 128, 257, 400), (32, 8, 112, 112, 128, 650), (32, 8, 112, 112, 127, 650),
                                               (32, 4, 96, 64, 512, 321), (32, 4, 96, 64, 511, 321), (32, 4, 64, 128, 256, 650), (33, 3, 65, 66, 300, 641)])
def test_on_both_sides_of_the_choice(gpu_ctx, H, G, d, dv, window, T):
    rng = np.random.default_rng(d + window)
    to = lambda x: torch.tensor(x).to(torch.bfloat16).double().numpy()
    q, k, v = (to(rng.standard_normal((T, n, e))) for n, e in ((H, d), (G, d), (G, dv)))
    r1, r2 = rng.random(H) + 0.2, rng.random(H) * 0.3
    want = F.window_attention(q, k, v, window, d ** -0.5, r1, r2).reshape(T, -1)
    got = run_window(S.SeqOps(gpu_ctx), q, k, v, window, d ** -0.5, r1, r2, torch.bfloat16, [T])
    gpu_ctx.check_status()
    assert rel(got, want) < 2 ** -8                      # as above


@pytest.mark.parametrize("H,d,sh,dv,window,cuts", [(2, 128, 64, 128, 2000, [643]), (2, 128, 64, 128, 130, [257, 3, 300]), (3, 120, 8, 104, 257, [129, 400]),
                                                   (2, 48, 16, 128, 300, [500]), (2, 184, 8, 64, 64, [64, 65, 200]), (1, 136, 0, 128, 1, [200]), (12, 64, 32, 64, 2, [700])])
def test_plain_rows_over_many_tiles(gpu_ctx, H, d, sh, dv, window, cuts):
    """Keys and values as rows, a part of every key shared by the heads; what a row does not see is not finite."""
    from hf2q_b200 import ops
    rng, T, sop = np.random.default_rng(d + window), sum(cuts), S.SeqOps(gpu_ctx)
    to = lambda *s: torch.tensor(rng.standard_normal(s)).to(torch.bfloat16)
    q, k, shared, v = 2 * to(T, H, d + sh), to(T, H, d), to(T, max(sh, 8)), to(T, H, dv)
    cap, at, outs, nan = window - 1 + max(cuts), 0, [], float("nan")
    ring = torch.full((cap, max(sh, 8)), nan, dtype=torch.bfloat16, device="cuda")
    for m in cuts:
        first = max(0, at - (window - 1))
        rows = torch.cat([x[first:at + m].reshape(at + m - first, -1) for x in (k, v)], 1)
        rows = torch.cat([rows, torch.full_like(rows[:3], nan)]).cuda().contiguous()
        ring[torch.arange(at, at + m, device="cuda") % cap] = shared[at:at + m].cuda()
        qd, out, pos = q[at:at + m].reshape(m, -1).cuda().contiguous(), torch.empty(m, H * dv, device="cuda"), torch.tensor([at], dtype=torch.int32, device="cuda")
        a = S.struct(S.WindowAttn, qkv=qd, k_cache=rows, v_cache=rows.data_ptr() + 2 * H * d, heads=H, kv_heads=H, dim=d, vdim=dv, window=window, capacity=cap,
                     cache_dtype=ops.DT_BF16, scale=(d + sh) ** -0.5, eps=1e-5, pos=pos, linear=1, row_stride=H * (d + dv), k_head_stride=d, v_head_stride=dv,
                     k_shared=ring if sh else None, shared_dim=sh, shared_stride=max(sh, 8), shared_capacity=cap)
        sop.window_prefill(a, m, qd, None, 0, out)
        outs.append(out)
        at += m
    gpu_ctx.check_status()
    keys = torch.cat([k.double(), shared.double()[:, None, :sh].expand(T, H, sh)], 2).transpose(0, 1)
    s = q.double().transpose(0, 1) @ keys.transpose(1, 2) * (d + sh) ** -0.5
    dist = torch.arange(T)[:, None] - torch.arange(T)[None]
    want = (torch.softmax(s.masked_fill((dist < 0) | (dist >= window), -float("inf")), -1) @ v.double().transpose(0, 1)).transpose(0, 1).reshape(T, -1)
    assert rel(torch.cat(outs), want.numpy()) < 2 ** -8
