"""A tensor-core product starts under the launch in front of it; its bounded waits do not count that launch's time."""
import pytest
import torch

import oracle
import hf2q_b200 as hq
from hf2q_b200 import ops, seqops as S
from tests.util import make_quant_weight

pytestmark = pytest.mark.gpu
DEV = "cuda"


# the forms whose weight ring is no deeper than the buffers it fills: 256 rows, and 128 in Q8_0
@pytest.mark.parametrize("t,m", [(oracle.Q4_0, 256), (oracle.Q8_0, 100)])
def test_behind_a_launch_of_more_than_the_limit(gpu_ctx, t, m):
    sop, n, k = S.SeqOps(gpu_ctx), 28672, 2048
    w = hq.load_quant_weight(gpu_ctx, make_quant_weight(t, n, k, seed=m), t, n, k)
    panel, want, got = torch.randn(m, k, device=DEV).half(), torch.empty(m, n, device=DEV), torch.zeros(m, n, device=DEV)

    def product(y):
        gpu_ctx._check(gpu_ctx._lib.hf2q_cuda_qmatmul_panel(gpu_ctx._h, gpu_ctx._stream(), panel.data_ptr(), ops.row_segments([w]), 1, None, y.data_ptr(), m, k))

    # a recurrence of one head, the same token again and again: a few CTAs, all on the chip at once, for as long as there are tokens
    row, gates = torch.randn(64, device=DEV), torch.zeros(1, device=DEV)
    state = [torch.zeros(8 * 32, device=DEV) for _ in range(3)]
    a = S.struct(S.MLstm, proj=row, ld=0, q_off=0, k_off=8, v_off=16, i_off=24, f_off=25, i_bias=gates, f_bias=gates, s=state[0], n=state[1], mx=state[2], heads=1,
                 dim=8, vdim=8, gate_cap=8.0)

    def ms(tokens, then):
        out, e0, e1 = torch.empty(tokens, 8, device=DEV), torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        sop.mlstm(a, tokens, out)
        then()
        e1.record()
        e1.synchronize()
        return e0.elapsed_time(e1)

    product(want)
    ms(1 << 16, lambda: None)
    tokens = int((1 << 18) * 1800 / ms(1 << 18, lambda: None))
    assert ms(tokens, lambda: product(got)) > 1300                # a wait gives up after 2^31 ticks, 1.1 s
    gpu_ctx.check_status()
    assert torch.equal(got, want)
