"""Tensor-core products whose K-blocks are shared by the CTAs of a cluster, with fewer, as many and more clusters than run side by side
with one CTA to an SM."""
import pytest
import torch

import oracle
import hf2q_b200 as hq
from hf2q_b200 import ops
from tests.util import make_quant_weight, rel_l2

pytestmark = pytest.mark.gpu
DEV = "cuda"


# rows of weights: clusters of four at up to 64 rows, of two beyond; 80 to 148 CTAs, or two to an SM of the pair
@pytest.mark.parametrize("n", [2560, 4096, 4096 + 16, 4608, 4736])
@pytest.mark.parametrize("m", [9, 33, 64, 65, 128])
def test_products(gpu_ctx, n, m):
    k, t = 2048, oracle.Q4_K
    g, u = (make_quant_weight(t, n, k, seed=s) for s in (0, 1))
    gate, up = hq.load_quant_weight(gpu_ctx, g, t, n, k), hq.load_quant_weight(gpu_ctx, u, t, n, k)
    x = torch.randn(m, k, generator=torch.Generator(device=DEV).manual_seed(n + m), device=DEV).half().float()      # (exact in the panel)
    gf, uf = (oracle.matmul_f64(x.cpu().numpy(), oracle.dequantize(t, w).reshape(n, k)) for w in (g, u))
    y, act = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    for _ in range(3):                                            # one behind the other, each started under the one in front
        ops.quantized_matmul_segments(gpu_ctx, x, [gate], y, m)
        ops.quantized_matmul_swiglu(gpu_ctx, x, gate, up, act, m)
    # f16 weights: 2^-11 each, k of them with random signs
    assert rel_l2(y.cpu().numpy(), gf) < 2 ** -11
    want = torch.from_numpy(gf)
    assert rel_l2(act.cpu().numpy(), (want * torch.sigmoid(want) * torch.from_numpy(uf)).numpy()) < 3 * 2 ** -11
    gpu_ctx.check_status()
