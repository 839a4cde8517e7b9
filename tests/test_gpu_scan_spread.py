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


# portions of one batch of tokens or several, of up to 8 tokens (one column a lane group) or more (two), on fewer or more CTAs than SMs
PORTIONS = [(6, 128, 128, 1), (32, 128, 128, 8), (32, 128, 128, 9), (150, 40, 9, 33), (19, 64, 130, 70), (3, 256, 33, 40), (16, 256, 256, 16), (20, 100, 128, 3)]


@pytest.mark.parametrize("heads,dim,vdim,m", PORTIONS)
def test_delta_portions(gpu_ctx, heads, dim, vdim, m):
    sop, g, kvh = S.SeqOps(gpu_ctx), torch.Generator(device=DEV).manual_seed(heads + m), heads if heads % 2 else heads // 2
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    unit = lambda x: x / x.norm(dim=-1, keepdim=True)
    q, k, v = unit(rand(m, kvh, dim)) * dim ** -0.5, unit(rand(m, kvh, dim)), rand(m, heads, vdim)
    qkv = torch.cat([x.reshape(m, -1) for x in (q, k, v)], 1).contiguous()
    beta, decay = torch.rand((m, heads), generator=g, device=DEV), torch.exp(-0.1 * torch.rand((m, heads, dim), generator=g, device=DEV))
    s = rand(heads, vdim, S.pad32(dim))
    s[..., dim:] = 0
    S0, out, one, pos = s[..., :dim].double(), torch.empty(m, heads * vdim, device=DEV), rand(heads * 8), torch.zeros(1, dtype=torch.int32, device=DEV)
    a = S.struct(S.Delta, proj=one, ld=8, q_conv=one, k_conv=one, v_conv=one, a_log=one, dt_bias=one, a2=one, g2=one, conv_state=one, s=s, pos=pos,
                 heads=heads, kv_heads=kvh, dim=dim, vdim=vdim, taps=4, a_rank_ld=8, g_rank_ld=8)
    sop.delta_scan(a, m, qkv, beta, decay, out)
    gpu_ctx.check_status()
    Q, K = (x.double().repeat_interleave(heads // kvh, 1) for x in (q, k))
    want = torch.empty(m, heads, vdim, dtype=torch.float64, device=DEV)
    for t in range(m):
        S0 = S0 * decay[t].double()[:, None]
        u = beta[t].double()[:, None] * (v[t].double() - torch.einsum("hvk,hk->hv", S0, K[t]))
        S0 = S0 + u[..., None] * K[t][:, None]
        want[t] = torch.einsum("hvk,hk->hv", S0, Q[t])
    bound = 2 ** -24 * (dim + m)                          # as above
    assert (out.view_as(want).double() - want).norm() < bound * want.norm()
    assert (s[..., :dim].double() - S0).norm() < bound * S0.norm()
    assert (s[..., dim:] == 0).all()


@pytest.mark.parametrize("heads,dim,vdim,m", PORTIONS)
def test_mlstm_portions(gpu_ctx, heads, dim, vdim, m):
    sop, g, cap = S.SeqOps(gpu_ctx), torch.Generator(device=DEV).manual_seed(heads + m), 15.0
    o, slices = heads * (2 * dim + vdim), -(-vdim // 16)
    proj = torch.randn((m, o + 2 * heads), generator=g, device=DEV)
    proj[:, heads * dim:2 * heads * dim] += 0.5           # (normalisers away from zero, where a quotient keeps no digits)
    proj[:, :heads * dim] += 0.5
    ib, fb = torch.randn(heads, generator=g, device=DEV), 3 + torch.randn(heads, generator=g, device=DEV)
    s, n, mx = torch.zeros(heads, vdim, S.pad32(dim), device=DEV), torch.zeros(heads, slices, S.pad32(dim), device=DEV), torch.zeros(heads, slices, device=DEV)
    out = torch.empty(m, heads * vdim, device=DEV)
    a = S.struct(S.MLstm, proj=proj, ld=proj.shape[1], q_off=0, k_off=heads * dim, v_off=2 * heads * dim, i_off=o, f_off=o + heads, i_bias=ib, f_bias=fb, s=s,
                 n=n, mx=mx, heads=heads, dim=dim, vdim=vdim, gate_cap=cap)
    sop.mlstm(a, m, out)
    gpu_ctx.check_status()
    P = proj.double()
    q, k, v = (P[:, i:j].view(m, heads, -1) for i, j in ((0, heads * dim), (heads * dim, 2 * heads * dim), (2 * heads * dim, o)))
    ig, fg = (cap * torch.tanh((P[:, i:i + heads] + b.double()) / cap) for i, b in ((o, ib), (o + heads, fb)))
    fg = -torch.nn.functional.softplus(-fg)
    S0, N, M = torch.zeros(heads, vdim, dim, dtype=torch.float64, device=DEV), torch.zeros(heads, dim, dtype=torch.float64, device=DEV), torch.zeros(heads, dtype=torch.float64, device=DEV)
    want = torch.empty(m, heads, vdim, dtype=torch.float64, device=DEV)
    for t in range(m):
        new = torch.maximum(fg[t] + M, ig[t])
        keep, write, M = torch.exp(fg[t] + M - new), torch.exp(ig[t] - new), new
        S0, N = keep[:, None, None] * S0 + (write[:, None] * v[t])[..., None] * k[t][:, None], keep[:, None] * N + write[:, None] * k[t]
        num, den = (torch.einsum(e, x, q[t]) * dim ** -0.5 for e, x in (("hvk,hk->hv", S0), ("hk,hk->h", N)))
        want[t] = num / (torch.maximum(den.abs(), torch.exp(-M)) + 1e-6)[:, None]
    bound = 2 ** -24 * (dim + 16 * m)                     # gate logarithms of up to 15 are carried in f32, over m tokens
    assert (s[..., :dim].double() - S0).norm() < bound * S0.norm()
    assert (out.view_as(want).double() - want).norm() < 4 * bound * want.norm()
    assert (n[..., :dim].double() - N[:, None]).norm() < bound * N.norm() * slices ** 0.5


# tokens of a CTA: 1 .. 16, by the size of the portion; the last CTA's share is shorter
@pytest.mark.parametrize("m,at", [(1, 5), (2, 0), (7, 3), (17, 1), (130, 2), (700, 0), (2100, 6)])
@pytest.mark.parametrize("heads,dim,vdim", [(2, 40, 24), (16, 128, 128), (6, 200, 300)])
def test_convolution_inputs(gpu_ctx, m, at, heads, dim, vdim):
    """delta_prep and ssd_prep behind `at` earlier tokens of a sequence (four taps)."""
    sop, g, kvh = S.SeqOps(gpu_ctx), torch.Generator(device=DEV).manual_seed(m + dim), heads // 2
    rand = lambda *s: torch.randn(s, generator=g, device=DEV)
    pos = torch.tensor([at], dtype=torch.int32, device=DEV)

    def ring(x):                                          # the last three inputs before `at`, column t % 4 of a channel
        st = torch.zeros(x.shape[1], 4, device=DEV)
        for t in range(max(0, at - 3), at):
            st[:, t % 4] = x[t]
        return st

    def conv(x, w, bias=0.0):
        ext = torch.cat([torch.zeros(3, x.shape[1], dtype=torch.float64, device=DEV), x.double()])
        y = sum(ext[j:j + len(x)] * w.double()[:, j] for j in range(4)) + bias
        return (y * torch.sigmoid(y))[at:]

    close = lambda got, want: (got.double() - want).norm() <= 1e-6 * want.norm()          # four products and a few functions in f32
    C1 = 2 * kvh * dim + heads * vdim
    x, low = rand(at + m, C1 + heads), rand(at + m, 16)
    proj, w = torch.cat([x, low], 1).contiguous(), rand(C1, 4)
    qkv, beta, a1, g1, one = rand(m, C1), rand(m, heads), rand(m, 8), rand(m, 8), rand(heads * dim)
    a = S.struct(S.Delta, proj=proj[at:], ld=proj.shape[1], q_off=0, k_off=kvh * dim, v_off=2 * kvh * dim, b_off=C1, a1_off=C1 + heads, g1_off=C1 + heads + 8,
                 q_conv=w, k_conv=w[kvh * dim:], v_conv=w[2 * kvh * dim:], a_log=one, dt_bias=one, a2=one, g2=one, conv_state=(st := ring(x[:, :C1])), s=one, pos=pos,
                 heads=heads, kv_heads=kvh, dim=dim, vdim=vdim, taps=4, a_rank_ld=8, g_rank_ld=8)
    sop.delta_prep(a, m, qkv, beta, a1, g1)
    y = conv(x[:, :C1], w)
    q, k = (y[:, i * kvh * dim:(i + 1) * kvh * dim].view(m, kvh, dim) for i in (0, 1))
    unit = lambda v: v / (v.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    assert close(qkv, torch.cat([(unit(q) * dim ** -0.5).reshape(m, -1), unit(k).reshape(m, -1), y[:, 2 * kvh * dim:]], 1))
    assert close(beta, torch.sigmoid(x[at:, C1:].double()))
    assert torch.equal(a1, low[at:, :8]) and torch.equal(g1, low[at:, 8:])
    C2 = heads * vdim + 2 * dim
    x, w, bias, dt_bias, a_log = rand(at + m, C2 + heads), rand(C2, 4), rand(C2), rand(heads), rand(heads)
    xbc, dt, la = rand(m, C2), rand(m, heads), rand(m, heads)
    b = S.struct(S.Ssd, proj=x[at:], ld=C2 + heads, off=0, conv=w, conv_bias=bias, dt_bias=dt_bias, a_log=a_log, d=one, conv_state=(st2 := ring(x[:, :C2])), s=one,
                 heads=heads, groups=1, state=dim, vdim=vdim, taps=4, pos=pos)
    sop.ssd_prep(b, m, xbc, dt, la)
    gpu_ctx.check_status()
    assert close(xbc, conv(x[:, :C2], w, bias.double()))
    steps = torch.nn.functional.softplus(x[at:, C2:].double() + dt_bias.double())
    assert close(dt, steps) and close(la, -torch.exp(a_log.double()) * steps)
