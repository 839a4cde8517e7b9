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
