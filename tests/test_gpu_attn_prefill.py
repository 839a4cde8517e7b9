"""Prompt attention over the 8-bit cache: the tensor-core kernel against softmax attention in 64 bits on the same codes."""
import ctypes as C

import pytest
import torch

from hf2q_b200 import _lib, decoder, ops

pytestmark = pytest.mark.gpu
HD = 128


def case(group, n_kv, pos0, m, k_scale, v_scale, growing, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    T, S = pos0 + m, pos0 + m + 3
    codes = [torch.randint(-127, 128, (n_kv, S, HD), generator=g, device="cuda", dtype=torch.int8) for _ in range(2)]
    scales = [s * (0.5 + torch.rand((n_kv, S), generator=g, device="cuda")) / 127 for s in (k_scale, v_scale)]
    if growing:                                          # scores grow with the position: the running maximum rises in every block
        scales[0] = scales[0] * torch.linspace(0.05, 4.0, S, device="cuda")
    scales[0][:, T:], scales[1][:, T:] = float("nan"), float("nan")          # what no row sees is not touched
    qkv = torch.randn((m, (group + 2) * n_kv * HD), generator=g, device="cuda") * HD ** -0.5
    return qkv, codes, scales, T, S


@pytest.mark.parametrize("group,n_kv,pos0,m,k_scale,v_scale,growing,dtype", [
    (4, 8, 0, 1, 1.0, 1.0, False, torch.float32),
    (4, 2, 0, 63, 1.0, 1.0, False, torch.float32),
    (4, 2, 0, 65, 2.0, 1.0, True, torch.float32),
    (8, 1, 5, 300, 2.0, 1.0, True, torch.bfloat16),
    (1, 3, 130, 257, 2.0, 1.0, True, torch.float32),
    (2, 2, 1000, 129, 1.0, 5e3, True, torch.float32),    # V scales at which the exponentials may not pass 1
    (4, 2, 4001, 97, 3.0, 1.0, False, torch.bfloat16),
    (1, 1, 64, 64, 1.0, 1e-4, False, torch.float32),
])
def test_prompt_attention_matches_softmax(gpu_ctx, group, n_kv, pos0, m, k_scale, v_scale, growing, dtype):
    qkv, codes, scales, T, S = case(group, n_kv, pos0, m, k_scale, v_scale, growing, seed=m)
    nq = group * n_kv
    kv = decoder._KvCache(codes[0].data_ptr(), scales[0].data_ptr(), codes[1].data_ptr(), scales[1].data_ptr(), n_kv, HD, S)
    out = torch.full((m, nq * HD), float("nan"), device="cuda", dtype=dtype)
    lib = _lib.load()
    gpu_ctx._check(lib.hf2q_cuda_attn_prefill(gpu_ctx._h, torch.cuda.current_stream().cuda_stream, qkv.data_ptr(), m, nq, C.byref(kv), pos0,
                                              out.data_ptr(), ops.DT_F32 if dtype == torch.float32 else ops.DT_BF16))
    gpu_ctx.check_status()
    k, v = ((c[:, :T].double() * s[:, :T, None].double()) for c, s in zip(codes, scales))
    q = qkv[:, :nq * HD].double().view(m, n_kv, group, HD)
    s = torch.einsum("tgrd,gpd->gtrp", q, k)
    hidden = torch.arange(T, device="cuda")[None] > pos0 + torch.arange(m, device="cuda")[:, None]
    want = torch.einsum("gtrp,gpd->tgrd", torch.softmax(s.masked_fill(hidden[None, :, None], -float("inf")), dim=-1), v).reshape(m, nq * HD)
    # probability * v_scale and q are f16: 2^-11 of the value each, the second times the spread of a score; bf16 results 2^-9 more
    spread = s.masked_fill(hidden[None, :, None], 0).std().item()
    bound = 2 ** -11 * (1 + spread) + (2 ** -9 if dtype == torch.bfloat16 else 0)
    err = (out.double() - want).norm() / want.norm()
    assert err < bound, (err.item(), bound)


def attend(ctx, qkv, codes, scales, S, m, nq, n_kv, pos0, out):
    kv = decoder._KvCache(codes[0].data_ptr(), scales[0].data_ptr(), codes[1].data_ptr(), scales[1].data_ptr(), n_kv, HD, S)
    ctx._check(_lib.load().hf2q_cuda_attn_prefill(ctx._h, torch.cuda.current_stream().cuda_stream, qkv.data_ptr(), m, nq, C.byref(kv), pos0, out.data_ptr(),
                                                  ops.DT_F32 if out.dtype == torch.float32 else ops.DT_BF16))


@pytest.mark.parametrize("pos0,m", [(0, 1500), (64, 700), (640, 2048)])
def test_waves_of_ctas_agree(gpu_ctx, pos0, m):
    """CTAs of all lengths (1 block to dozens) side by side and in several waves, many times: every wait ends, every run has the same bits."""
    qkv, codes, scales, T, S = case(4, 8, pos0, m, 2.0, 1.0, True, seed=m)
    first, again = (torch.full((m, 32 * HD), float("nan"), device="cuda") for _ in range(2))
    attend(gpu_ctx, qkv, codes, scales, S, m, 32, 8, pos0, first)
    for _ in range(40):
        attend(gpu_ctx, qkv, codes, scales, S, m, 32, 8, pos0, again)
        assert torch.equal(first, again)
    gpu_ctx.check_status()
    assert first.isfinite().all()


@pytest.mark.parametrize("group,m", [(1, 1), (1, 127), (1, 129), (1, 161), (2, 65), (4, 7), (4, 33), (8, 1), (8, 17)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shift", [0, 1])
def test_tiles_that_end_inside_a_warp(gpu_ctx, group, m, dtype, shift):
    """Rows past the last token share a warp with live ones: live rows come whole, aligned or not, and nothing else is written."""
    qkv, codes, scales, T, S = case(group, 2, 70, m, 2.0, 1.0, True, seed=m)
    nq = 2 * group
    flat = torch.full((shift + (m + 3) * nq * HD,), -7.0, device="cuda", dtype=dtype)
    out = flat[shift:shift + m * nq * HD].view(m, nq * HD)
    whole = torch.empty((m + 128, nq * HD), device="cuda", dtype=dtype)[:m]
    attend(gpu_ctx, qkv, codes, scales, S, m, nq, 2, 70, whole)
    attend(gpu_ctx, qkv, codes, scales, S, m, nq, 2, 70, out)
    gpu_ctx.check_status()
    k, v = ((c[:, :T].double() * s[:, :T, None].double()) for c, s in zip(codes, scales))
    q = qkv[:, :nq * HD].double().view(m, 2, group, HD)
    s = torch.einsum("tgrd,gpd->gtrp", q, k)
    hidden = torch.arange(T, device="cuda")[None] > 70 + torch.arange(m, device="cuda")[:, None]
    want = torch.einsum("gtrp,gpd->tgrd", torch.softmax(s.masked_fill(hidden[None, :, None], -float("inf")), dim=-1), v).reshape(m, nq * HD)
    spread = s.masked_fill(hidden[None, :, None], 0).std().item()
    bound = 2 ** -11 * (1 + spread) + (2 ** -9 if dtype == torch.bfloat16 else 0)        # as above
    row_err = (out.double() - want).norm(dim=1) / want.norm(dim=1)
    assert row_err.max() < 4 * bound                     # a row alone: no averaging over rows
    assert torch.equal(out, whole)
    assert (flat[:shift] == -7).all() and (flat[shift + m * nq * HD:] == -7).all()


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("pos0,m,at", [(0, 200, 77), (30, 129, 30 + 128), (64, 100, 64 + 1)])
def test_hidden_scales_do_not_reach_a_row(gpu_ctx, bad, which, pos0, m, at):
    """A K or V scale that is not finite shows in the rows that see its position and in no other of the tile."""
    qkv, codes, scales, T, S = case(2, 2, pos0, m, 2.0, 1.0, True, seed=m)
    clean = [s.clone() for s in scales]
    scales[which][:, at] = bad
    out = torch.empty((m, 4 * HD), device="cuda")
    attend(gpu_ctx, qkv, codes, scales, S, m, 4, 2, pos0, out)
    gpu_ctx.check_status()
    k, v = ((c[:, :T].double() * s[:, :T, None].double()) for c, s in zip(codes, clean))
    s = torch.einsum("tgrd,gpd->gtrp", qkv[:, :4 * HD].double().view(m, 2, 2, HD), k)
    hidden = torch.arange(T, device="cuda")[None] > pos0 + torch.arange(m, device="cuda")[:, None]
    want = torch.einsum("gtrp,gpd->tgrd", torch.softmax(s.masked_fill(hidden[None, :, None], -float("inf")), dim=-1), v).reshape(m, 4 * HD)
    n = at - pos0                                        # the first row that sees the position
    bound = 2 ** -11 * (1 + s.masked_fill(hidden[None, :, None], 0).std().item())
    assert (out[:n].double() - want[:n]).norm() < bound * want[:n].norm()
    if which == 1:
        assert not out[n].isfinite().any()


@pytest.mark.parametrize("group,n_kv,pos0,m", [(1, 3, 0, 1), (2, 2, 7, 1), (4, 8, 0, 33), (8, 1, 40, 8), (4, 2, 0, 48), (8, 2, 1, 47), (1, 2, 0, 49), (2, 1, 47, 2)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_few_positions(gpu_ctx, group, n_kv, pos0, m, dtype):
    """Up to 48 positions in all a kernel in f32, above that the tensor cores; infinite scales of later tokens reach no row."""
    qkv, codes, scales, T, S = case(group, n_kv, pos0, m, 3.0, 1.0, True, seed=m)
    clean, nq = [s.clone() for s in scales], group * n_kv
    if m > 1:
        scales[0][:, T - 1], scales[1][:, T - 1] = float("nan"), float("inf")
    out = torch.full((m, nq * HD), float("nan"), device="cuda", dtype=dtype)
    attend(gpu_ctx, qkv, codes, scales, S, m, nq, n_kv, pos0, out)
    gpu_ctx.check_status()
    k, v = ((c[:, :T].double() * s[:, :T, None].double()) for c, s in zip(codes, clean))
    s = torch.einsum("tgrd,gpd->gtrp", qkv[:, :nq * HD].double().view(m, n_kv, group, HD), k)
    hidden = torch.arange(T, device="cuda")[None] > pos0 + torch.arange(m, device="cuda")[:, None]
    want = torch.einsum("gtrp,gpd->tgrd", torch.softmax(s.masked_fill(hidden[None, :, None], -float("inf")), dim=-1), v).reshape(m, nq * HD)
    spread, n = s.masked_fill(hidden[None, :, None], 0).abs().max().item(), max(m - 1, 1)
    bound = (2 ** -23 * (12 + spread) if T <= 48 else 2 ** -11 * (1 + spread)) + (2 ** -9 if dtype == torch.bfloat16 else 0)     # sums of 128 terms; a score's error is its size's
    assert (out[:n].double() - want[:n]).norm() < bound * want[:n].norm()
