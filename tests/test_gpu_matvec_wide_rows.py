"""One-row products behind rows that are too long for the registers of their prologue: whole 16-byte groups, ragged and unaligned ones."""
import numpy as np
import pytest
import torch

from hf2q_b200 import seqops as S

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("width,off", [(4612, 0), (5120, 0), (8192, 0), (5121, 0), (4624, 1)])
@pytest.mark.parametrize("shift", [False, True])
@pytest.mark.parametrize("pos", [6, 7])
def test_norm_prologue(gpu_ctx, width, off, shift, pos):
    """off: the norm starts off a 16-byte boundary."""
    sop, rng, n, k = S.SeqOps(gpu_ctx), np.random.default_rng(width + pos), 200, S.pad8(width)
    f = lambda *s: torch.from_numpy(rng.standard_normal(s).astype(np.float32)).to(DEV)
    w = S.DenseWeight(torch.from_numpy(rng.standard_normal((n, width)) / width ** 0.5).to(torch.bfloat16), DEV)
    x, norm, mu, state, x_out, y = f(width), f(width + off)[off:], f(width), f(2, width), torch.zeros(width, device=DEV), torch.zeros(n, device=DEV)
    was, at = state.clone(), torch.tensor([pos], dtype=torch.int32, device=DEV)
    p = S.struct(S.PreNorm, x=x, x_out=x_out, norm=norm, eps=1e-5, width=width, **(dict(shift=mu, shift_state=state, pos=at) if shift else {}))
    seg = S.struct(S.Matvec, w=w.w, y=y, n=n, k=k)
    seg.pre = p
    try:
        sop.matvec(S.PRO_NORM, seg)
    except Exception:
        assert off, "only an unaligned row may be refused"
        return
    gpu_ctx.check_status()
    d = lambda t: t.double()
    h = d(x) * torch.rsqrt((d(x) ** 2).mean() + 1e-5) * d(norm)
    row, want_state = h, d(was)
    if shift:
        want_state[pos & 1] = h
        row = h + (d(was[(pos + 1) & 1]) - h) * d(mu)
    assert torch.equal(x_out, x)
    assert (d(state) - want_state).abs().max() <= 8 * 2 ** -23 * h.abs().max()
    want, size = d(w.w[:, :width]) @ row, d(w.w[:, :width]).abs() @ row.abs()
    # f32 sums of k products in any order, and a root, three products and two sums in front of them
    assert ((d(y) - want).abs() <= (64 + 16) * 2 ** -24 * size).all()


# held in registers up to 9216: spans of 128 shared by a head, one head of more than 64 of them; beyond, and heads of other lengths, not held
@pytest.mark.parametrize("heads,dim", [(37, 128), (40, 128), (64, 128), (18, 512), (1, 8320), (1, 9216), (73, 128), (50, 120)])
@pytest.mark.parametrize("kind", [S.GATE_SIGMOID_LAST, S.GATE_SILU_FIRST])
def test_gated_prologue(gpu_ctx, heads, dim, kind):
    sop, g, n, width = S.SeqOps(gpu_ctx), torch.Generator(device=DEV).manual_seed(heads * dim), 150, heads * dim
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)
    w = S.DenseWeight((r(n, width) / width ** 0.5).to(torch.bfloat16).cpu(), DEV)
    o, gate, norm, y = r(width), r(width), r(width), torch.zeros(n, device=DEV)
    seg = S.struct(S.Matvec, w=w.w, y=y, n=n, k=w.k)
    seg.gated = S.struct(S.GatedHeads, o=o, gate=gate, norm=norm, ldo=width, ldg=width, heads=heads, head_dim=dim, norm_all=1, eps=1e-5, kind=kind)
    sop.matvec(S.PRO_GATED, seg)
    gpu_ctx.check_status()
    o, gate, norm = (t.double().view(heads, dim) for t in (o, gate, norm))
    if kind == S.GATE_SILU_FIRST:
        o = o * gate * torch.sigmoid(gate)
    h = o * torch.rsqrt((o * o).mean(1, keepdim=True) + 1e-5) * norm
    row = (h if kind == S.GATE_SILU_FIRST else h * torch.sigmoid(gate)).flatten()
    m = w.w[:, :width].double()
    # as above, with a sigmoid and its product
    assert ((y.double() - m @ row).abs() <= (64 + 32) * 2 ** -24 * (m.abs() @ row.abs())).all()
