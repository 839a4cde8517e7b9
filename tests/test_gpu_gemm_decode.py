"""The 32-element formats in the tensor-core product: one-hot rows give back the weights, rounded to f16 once."""
import numpy as np
import pytest
import torch

import hf2q_b200 as hq
import oracle
from tests.util import make_quant_weight, random_finite_blocks

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = hq.GpuContext(0)
    yield c
    c.close()


@pytest.mark.parametrize("ggml_type", [2, 8])
@pytest.mark.parametrize("random_bits", [False, True])
@pytest.mark.parametrize("n,k", [(1, 256), (130, 512), (65, 2304)])
def test_one_hot_rows(ctx, ggml_type, random_bits, n, k):
    raw = random_finite_blocks(ggml_type, n * k // 32, seed=n) if random_bits else make_quant_weight(ggml_type, n, k, seed=n)
    raw = np.ascontiguousarray(raw).reshape(n * k // 32, -1)
    raw[:, 1] &= 0xBF                                       # scales below 2: every weight fits f16 (subnormal scales stay)
    raw = raw.reshape(-1)
    w = hq.load_quant_weight(ctx, raw, ggml_type, n, k)
    x, y = torch.eye(k, device="cuda"), torch.empty((k, n), device="cuda")
    hq.quantized_matmul_ggml(ctx, x, w, y, w.matmul_params(k))
    ctx.check_status()
    want = oracle.dequantize(ggml_type, raw).reshape(n, k).astype(np.float16)
    assert np.array_equal(y.cpu().numpy().T, want.astype(np.float32))


# few rows: the K-blocks (256 columns) of a tile are shared by 1, 2, 4 or 8 CTAs, unevenly where they do not divide; 512 columns
# are never shared, 2560 x 256 rows hardly
@pytest.mark.parametrize("ggml_type", [8, 12, 14])
@pytest.mark.parametrize("m,n,k", [(9, 1, 512), (9, 130, 1024), (37, 200, 2304), (64, 64, 4352), (65, 129, 4352), (128, 2560, 2304), (260, 300, 2304),
                                   (600, 1100, 1280)])
def test_shared_k_blocks(ctx, ggml_type, m, n, k):
    from hf2q_b200 import ops
    k = -(-k // 2048) * 2048 if ggml_type == 14 else k      # Q6_K rows of other lengths take another kernel
    raw = [make_quant_weight(ggml_type, n, k, seed=s) for s in (n, n + 1)]
    gate, up = (hq.load_quant_weight(ctx, r, ggml_type, n, k) for r in raw)
    g = torch.Generator().manual_seed(m)
    x, res = torch.randn((m, k), generator=g), torch.randn((m, n), generator=g).cuda()
    y, z, act, both = (torch.full((m, n), float("nan"), device="cuda") for _ in range(4))
    ops.quantized_matmul_ggml(ctx, x.cuda(), gate, y, gate.matmul_params(m))
    ops.quantized_matmul_add(ctx, x.cuda(), gate, res, z, m)
    ops.quantized_matmul_ggml(ctx, x.cuda(), up, act, up.matmul_params(m))
    ops.quantized_matmul_swiglu(ctx, x.cuda(), gate, up, both, m)
    ctx.check_status()
    want = x.double().numpy() @ oracle.dequantize(ggml_type, raw[0]).reshape(n, k).astype(np.float64).T
    # both operands rounded to f16: 2^-11 of each product at most, added up at random
    assert np.linalg.norm(y.cpu().numpy() - want) < 1e-3 * np.linalg.norm(want)
    assert torch.equal(z, y + res)
    silu = torch.empty_like(y)
    ctx._check(ctx._lib.hf2q_cuda_silu_mul(ctx._h, ctx._stream(), y.data_ptr(), act.data_ptr(), silu.data_ptr(), y.numel()))
    assert torch.equal(both, silu)


# products whose shares come as one or two CTAs an SM, in tiles of 64 or 128 tokens
@pytest.mark.parametrize("ggml_type", [8, 13, 14])
@pytest.mark.parametrize("m,n,k", [(33, 6144, 2048), (64, 6144, 2048), (100, 4096, 2048), (128, 4000, 2048), (300, 1024, 2048), (1000, 512, 2048)])
def test_shares_of_wide_products(ctx, ggml_type, m, n, k):
    test_shared_k_blocks(ctx, ggml_type, m, n, k)


@pytest.mark.parametrize("m", [9, 130, 2500])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_activations_off_a_vector_boundary(ctx, m, dtype):
    n, k = 64, 512
    w = hq.load_quant_weight(ctx, make_quant_weight(12, n, k, seed=1), 12, n, k)
    flat = torch.randn(m * k + 1, generator=torch.Generator().manual_seed(m)).to(dtype).cuda()
    y, z = torch.empty((m, n), device="cuda"), torch.empty((m, n), device="cuda")
    hq.quantized_matmul_ggml(ctx, flat[1:].view(m, k), w, y, w.matmul_params(m))
    hq.quantized_matmul_ggml(ctx, flat[1:].clone().view(m, k), w, z, w.matmul_params(m))
    ctx.check_status()
    assert torch.equal(y, z) and y.isfinite().all()
