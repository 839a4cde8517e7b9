"""The state-space scan over more heads than the chip has SMs: how many CTAs share an SM must not show in the result."""
import pytest
import torch

from hf2q_b200 import seqops as S

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("heads,state,vdim,m", [(149, 32, 32, 33), (300, 16, 33, 70), (297, 256, 5, 31), (1000, 8, 64, 64)])
def test_many_heads(gpu_ctx, heads, state, vdim, m):
    sop, g = S.SeqOps(gpu_ctx), torch.Generator(device=DEV).manual_seed(heads)
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    channels = heads * vdim + 2 * state
    xbc, dt, d = rand(m, channels), torch.rand((m, heads), generator=g, device=DEV), rand(heads)
    la, proj, one = -dt * (0.5 + torch.rand(heads, generator=g, device=DEV)), rand(m, channels + heads), rand(channels * 4)
    s = rand(heads, vdim, S.pad32(state))
    s[..., state:] = 0
    S0, y = s[..., :state].double(), torch.empty(m, heads * vdim, device=DEV)
    conv_state, pos = torch.zeros(channels, 4, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    a = S.struct(S.Ssd, proj=proj, ld=channels + heads, off=0, conv=one, conv_bias=one, dt_bias=one, a_log=one, d=d, conv_state=conv_state, s=s, heads=heads,
                 groups=1, state=state, vdim=vdim, taps=4, pos=pos)
    sop.ssd_scan(a, m, xbc, dt, la, y)
    gpu_ctx.check_status()
    x, B, C = xbc.double().split([heads * vdim, state, state], dim=1)
    x, want = x.view(m, heads, vdim), torch.empty(m, heads, vdim, dtype=torch.float64, device=DEV)
    for t in range(m):
        S0 = S0 * torch.exp(la[t].double())[:, None, None] + (dt[t].double()[:, None] * x[t])[..., None] * B[t]
        want[t] = S0 @ C[t] + d.double()[:, None] * x[t]
    # 32-bit sums of `state` terms, carried over m tokens
    bound = 2 ** -24 * (state + m)
    assert (y.view_as(want).double() - want).norm() < bound * want.norm()
    assert (s[..., :state].double() - S0).norm() < bound * S0.norm()
