"""Panels: what the entries in front of a tensor-core product write is what the product's own conversion makes of their f32 results,
bit for bit."""
import ctypes as C

import pytest
import torch

import oracle
import hf2q_b200 as hq
from hf2q_b200 import decoder, ops
from tests.util import make_quant_weight

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _r(seed, *s):
    return torch.randn(*s, generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV)


# rows of whole 16-byte groups up to 8192 stay in registers; others, and unaligned ones, take the other kernel
@pytest.mark.parametrize("h", [4, 1020, 1024, 4096, 8192, 8196, 515])
@pytest.mark.parametrize("m", [1, 5])
@pytest.mark.parametrize("delta", [False, True])
def test_rms_norm(gpu_ctx, h, m, delta):
    lib, x, w, d = gpu_ctx._lib, 3.0 * _r(h, m, h), _r(h + 1, h), _r(h + 2, m, h) if delta else None
    want_x = x.double() + d.double() if delta else x.double()
    want = want_x * torch.rsqrt((want_x * want_x).mean(1, keepdim=True) + 1e-5) * w.double()
    outs = {}
    for dt in (torch.float32, torch.bfloat16, torch.float16):
        xx, out = x.clone(), torch.empty(m, h, dtype=dt, device=DEV)
        args = (gpu_ctx._h, gpu_ctx._stream(), xx.data_ptr(), d.data_ptr() if delta else None, w.data_ptr(), 1e-5, out.data_ptr())
        gpu_ctx._check(lib.hf2q_cuda_rms_norm_panel(*args, m, h) if dt == torch.float16 else lib.hf2q_cuda_rms_norm(*args, ops._TORCH_DT[dt], m, h))
        assert (xx.double() - want_x).abs().max() <= 2 ** -24 * want_x.abs().max()
        outs[dt] = out
    # a sum of h squares, a root, two products
    assert ((outs[torch.float32].double() - want).abs() <= 8 * 2 ** -23 * want.abs() + 1e-30).all()
    for dt in (torch.bfloat16, torch.float16):
        assert torch.equal(outs[dt], outs[torch.float32].to(dt))
    gpu_ctx.check_status()


def test_values_beyond_f16_are_clipped_and_noted(gpu_ctx):
    x, w, out = torch.zeros(1, 256, device=DEV), torch.full((256,), 1e6, device=DEV), torch.empty(1, 256, dtype=torch.float16, device=DEV)
    x[0, 3], x[0, 7] = 1.0, -1.0
    gpu_ctx._check(gpu_ctx._lib.hf2q_cuda_rms_norm_panel(gpu_ctx._h, gpu_ctx._stream(), x.data_ptr(), None, w.data_ptr(), 1e-5, out.data_ptr(), 1, 256))
    with pytest.raises(hq.Hf2qError):
        gpu_ctx.check_status()
    assert float(out[0, 3]) == 65504.0 and float(out[0, 7]) == -65504.0


# shared K-blocks in a cluster (few rows), one tile, ragged tiles of 64, 128 and 256 tokens
@pytest.mark.parametrize("t", [oracle.Q4_0, oracle.Q8_0, oracle.Q4_K, oracle.Q5_K, oracle.Q6_K])
@pytest.mark.parametrize("m", [9, 37, 65, 130, 600])
def test_products_on_panels(gpu_ctx, t, m):
    lib, n, k = gpu_ctx._lib, 1024 + 16, 2048
    w = [hq.load_quant_weight(gpu_ctx, make_quant_weight(t, r, c, seed=s), t, r, c) for s, (r, c) in enumerate([(n, k), (n, k), (96, k)])]
    x, f32 = _r(m, m, k), lambda c: torch.empty(m, c, device=DEV)
    panel = x.half()
    act, act16 = f32(n), torch.empty(m, n, dtype=torch.float16, device=DEV)
    ops.quantized_matmul_swiglu(gpu_ctx, x, w[0], w[1], act, m)
    ws = torch.empty(2 * m * k + 256, dtype=torch.uint8, device=DEV)
    for src, ws_ptr in ((panel, None), (x, (ws.data_ptr() + 255) // 256 * 256)):
        act16.fill_(7.0)
        gpu_ctx._check(lib.hf2q_cuda_qmatmul_swiglu_panel(gpu_ctx._h, gpu_ctx._stream(), src.data_ptr(), ops._TORCH_DT[src.dtype], w[0].ptr, w[1].ptr, act16.data_ptr(), m, n,
                                                          k, t, ws_ptr, 2 * m * k if ws_ptr else 0))
        assert torch.equal(act16, act.half())
    both, got = f32(n + 96), f32(n + 96)
    ops.quantized_matmul_segments(gpu_ctx, x, [w[0], w[2]], both, m)
    gpu_ctx._check(lib.hf2q_cuda_qmatmul_panel(gpu_ctx._h, gpu_ctx._stream(), panel.data_ptr(), ops.row_segments([w[0], w[2]]), 2, None, got.data_ptr(), m, k))
    assert torch.equal(got, both)
    res, one, add = _r(m + 1, m, n), f32(n), f32(n)
    ops.quantized_matmul_add(gpu_ctx, x, w[0], res, add, m)
    one.copy_(res)                                                # in place on the residual
    gpu_ctx._check(lib.hf2q_cuda_qmatmul_panel(gpu_ctx._h, gpu_ctx._stream(), panel.data_ptr(), ops.row_segments([w[0]]), 1, one.data_ptr(), one.data_ptr(), m, k))
    assert torch.equal(one, add)
    gpu_ctx.check_status()


@pytest.mark.parametrize("m,pos0", [(20, 0), (200, 0), (130, 300)])
@pytest.mark.parametrize("G", [1, 4])
def test_attention_writes_a_panel(gpu_ctx, m, pos0, G):
    n_kv, T = 2, pos0 + m
    codes = [torch.randint(-127, 128, (n_kv, T, 128), device=DEV, dtype=torch.int8) for _ in range(2)]
    scales = [(0.5 + torch.rand(n_kv, T, device=DEV)) / 127 for _ in range(2)]
    kv = decoder._KvCache(codes[0].data_ptr(), scales[0].data_ptr(), codes[1].data_ptr(), scales[1].data_ptr(), n_kv, 128, T)
    nq = G * n_kv
    qkv, out, panel = _r(m, m, (nq + 2 * n_kv) * 128) * 128 ** -0.5, torch.empty(m, nq * 128, device=DEV), torch.empty(m, nq * 128, dtype=torch.float16, device=DEV)
    args = (gpu_ctx._h, gpu_ctx._stream(), qkv.data_ptr(), m, nq, C.byref(kv), pos0)
    gpu_ctx._check(gpu_ctx._lib.hf2q_cuda_attn_prefill(*args, out.data_ptr(), ops.DT_F32))
    gpu_ctx._check(gpu_ctx._lib.hf2q_cuda_attn_prefill_panel(*args, panel.data_ptr()))
    assert torch.equal(panel, out.half())
    with pytest.raises(hq.Hf2qError):                             # the plain entry takes f32 and bf16 outputs, as before
        gpu_ctx._check(gpu_ctx._lib.hf2q_cuda_attn_prefill(*args, panel.data_ptr(), ops.DT_F16))
    gpu_ctx.check_status()


@pytest.mark.parametrize("n_q,n_kv,shift", [(8, 2, 0), (3, 3, 0), (8, 2, 1)])
def test_rotary_and_append(gpu_ctx, n_q, n_kv, shift):
    """shift: rows off 16-byte boundaries."""
    m, pos0, theta, S = 21, 5, 10000.0, 64
    heads = n_q + 2 * n_kv
    buf = _r(n_q, m * heads * 128 + shift)
    qkv = buf[shift:].view(m, heads, 128)
    src = qkv.double().clone()
    kc, vc = (torch.zeros(n_kv, S, 128, dtype=torch.int8, device=DEV) for _ in range(2))
    ks, vs = (torch.zeros(n_kv, S, device=DEV) for _ in range(2))
    kv, pos = decoder._KvCache(kc.data_ptr(), ks.data_ptr(), vc.data_ptr(), vs.data_ptr(), n_kv, 128, S), torch.tensor([pos0], dtype=torch.int32, device=DEV)
    gpu_ctx._check(gpu_ctx._lib.hf2q_cuda_rope_kv_append(gpu_ctx._h, gpu_ctx._stream(), qkv.data_ptr(), m, n_q, theta, pos.data_ptr(), C.byref(kv)))
    gpu_ctx.check_status()
    a = (torch.arange(m, device=DEV).double() + pos0)[:, None] * theta ** (-torch.arange(0, 128, 2, device=DEV).double() / 128)
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = src[..., 0::2], src[..., 1::2]
    turned = torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    # the angle itself, up to 26, is rounded in f32
    tol = 26 * 2 ** -22 * float(src.abs().max())
    assert (qkv[:, :n_q].double() - turned[:, :n_q] / 128 ** 0.5).abs().max() < tol
    for codes, scale, want in ((kc, ks, turned[:, n_q:n_q + n_kv]), (vc, vs, src[:, n_q + n_kv:])):
        sc = scale[:, pos0:pos0 + m].T[..., None].double()
        assert ((codes[:, pos0:pos0 + m].transpose(0, 1).double() * sc - want).abs() <= 0.5 * sc + tol).all()
        assert int(codes[:, :pos0].abs().sum()) == 0 and int(codes[:, pos0 + m:].abs().sum()) == 0
