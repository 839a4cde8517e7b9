"""One-row products against f64: rows of one piece and of many, a place of its own for every warp and none, row prologues at the edges of
what is held in registers."""
import numpy as np
import pytest
import torch

from hf2q_b200 import seqops as S
from oracle import fomatar_forward as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def sop(gpu_ctx):
    return S.SeqOps(gpu_ctx)


def f32(a):
    return torch.tensor(np.asarray(a), dtype=torch.float32, device=DEV)


def weight(n, k, seed):
    return S.DenseWeight((torch.randn(n, k, generator=torch.Generator().manual_seed(seed)) / k ** 0.5).to(torch.bfloat16), DEV)


def close(got, x, w, extra=0.0):
    """A term meets at most 44 roundings: 8 in its lane's group, 2 + 5 in the warp, one per piece (27), 2 for bias and residual."""
    w = w.w.cpu().double().numpy()[:, :x.size]
    got = got.detach().cpu().double().numpy().reshape(-1)
    bound = 44 * 2.0 ** -24 * (np.abs(w) @ np.abs(x) + np.abs(extra))
    assert (np.abs(got - (w @ x + extra)) <= bound).all()


# (pieces: 1, 1, 1, 2, 3, 5, 6, 9, 16, 17, 27; 150 rows leave CTAs without a row, 2500 give up to 17 to each)
@pytest.mark.parametrize("k", [8, 1016, 1024, 1032, 2056, 4104, 6144, 9208, 16384, 16392, 27648])
@pytest.mark.parametrize("n", [1, 150, 2500])
def test_pieces(sop, k, n):
    x = np.random.default_rng(k + n).standard_normal(k).astype(np.float32)
    w, xg, y = weight(n, k, k + n), f32(x), torch.full((1, n), 9.0, device=DEV)
    bias, res = torch.randn(n, device=DEV), torch.randn(1, n, device=DEV)
    sop.matvec(S.PRO_NONE, S.struct(S.Matvec, w=w.w, y=y, x=xg, bias=bias, residual=res, n=n, k=k, epilogue=S.EPI_ADD))
    close(y, x.astype(np.float64), w, (bias + res[0]).cpu().double().numpy())
    if n % 2 == 0:                                                          # rows in pairs: silu(gate) * up
        g = torch.empty((1, n // 2), device=DEV)
        sop.matvec(S.PRO_NONE, S.struct(S.Matvec, w=w.w, y=g, x=xg, n=n, k=k, epilogue=S.EPI_SWIGLU))
        v = w.w.cpu().double().numpy() @ x.astype(np.float64)
        want = v[0::2] * F.sigmoid(v[0::2]) * v[1::2]
        assert np.linalg.norm(g.cpu().double().numpy()[0] - want) < 1e-5 * np.linalg.norm(want)
    sop.ctx.check_status()


@pytest.mark.parametrize("width", [4, 2044, 2048, 2052, 4096, 4100, 6148])
@pytest.mark.parametrize("parts", [0, 1, 5])
def test_stream_prologue(sop, width, parts):
    rng, streams, n, eps = np.random.default_rng(width + parts), 4, 300, 1e-5
    x, c_in, norm = rng.standard_normal((streams, width)), rng.standard_normal(streams), rng.standard_normal(width)
    mix, gain, y = rng.standard_normal((streams, streams)), rng.standard_normal(streams), rng.standard_normal((max(parts, 1), width))
    new = mix.T @ x + gain[:, None] * y.sum(0) if parts else x
    h = F.rms((c_in @ new)[None], eps)[0] * norm
    w, out, x_out = weight(n, S.pad8(width), width), torch.zeros(1, n, device=DEV), torch.zeros(streams, width, device=DEV)
    t = dict(x=f32(x), c_in=f32(c_in), norm=f32(norm))
    if parts:
        t |= dict(y=f32(y), mix=f32(mix), out=f32(gain), x_out=x_out)
    p = S.struct(S.Hyper, x_streams=streams, streams=streams, width=width, y_parts=parts or None, eps=eps, **t)
    sop.matvec(S.PRO_HYPER, S.struct(S.Matvec, w=w.w, y=out, hyper=p, n=n, k=w.k))
    want = w.w.cpu().double().numpy()[:, :width] @ h
    assert np.linalg.norm(out.cpu().double().numpy()[0] - want) < 2e-5 * np.linalg.norm(want)
    assert not parts or np.linalg.norm(x_out.cpu().double().numpy() - new) < 2e-6 * np.linalg.norm(new)


# (down's row: top x pieces of ff)
@pytest.mark.parametrize("width,ff,experts,top", [(2048, 512, 8, 5), (1032, 1032, 4, 4), (2056, 8, 20, 17), (64, 2056, 6, 6)])
def test_expert_step(sop, width, ff, experts, top):
    rng = np.random.default_rng(width + ff)
    gu, down = weight(experts * 2 * ff, width, ff), weight(experts * width, ff, ff + 1)
    logits, h = rng.standard_normal(experts), rng.standard_normal(width).astype(np.float32)
    ids, act, y = torch.zeros(1, top, dtype=torch.int32, device=DEV), torch.zeros(top, ff, device=DEV), torch.zeros(1, width, device=DEV)
    keep = f32(logits), f32(h)
    sop.expert_step(S.struct(S.ExpertStep, gate_up=gu.w, down=down.w, logits=keep[0], h=keep[1], ids=ids, act=act, y=y, experts=experts, top=top, ff=ff,
                             width=width, k_in=width))
    score = F.sigmoid(logits.astype(np.float32).astype(np.float64))
    chosen = np.argsort(-score, kind="stable")[:top]
    assert ids.cpu().numpy()[0].tolist() == chosen.tolist()
    g = gu.w.cpu().double().numpy().reshape(experts, 2 * ff, width) @ h.astype(np.float64)
    d, want = down.w.cpu().double().numpy().reshape(experts, width, ff), 0.0
    for e in chosen:
        a, b = score[e] * g[e, 0::2], score[e] * g[e, 1::2]
        want = want + d[e] @ (a * F.sigmoid(a) * b)
    assert np.linalg.norm(y.cpu().double().numpy()[0] - want) < 1e-5 * np.linalg.norm(want)
    sop.ctx.check_status()


@pytest.mark.parametrize("heads,dim", [(1, 128), (3, 128), (16, 128), (8, 512), (36, 128), (37, 128), (5, 384), (6, 120)])
@pytest.mark.parametrize("kind,norm", [(S.GATE_SILU_FIRST, 1), (S.GATE_SIGMOID_LAST, 1), (S.GATE_SIGMOID_LAST, 0), (S.GATE_SIGMOID_LAST, None)])
def test_gated_prologue(sop, heads, dim, kind, norm):
    rng, n, k, eps = np.random.default_rng(heads * dim), 200, heads * dim, 1e-5
    o, gate, w = rng.standard_normal(k), rng.standard_normal(k), rng.standard_normal(k if norm != 0 else dim)
    v = (o * gate * F.sigmoid(gate) if kind == S.GATE_SILU_FIRST else o).reshape(heads, dim)
    if norm is not None:
        v = F.rms(v, eps) * w.reshape(-1, dim)
    v = v.reshape(-1) * (F.sigmoid(gate) if kind == S.GATE_SIGMOID_LAST else 1.0)
    t = dict(o=f32(o), gate=f32(gate)) | ({} if norm is None else dict(norm=f32(w)))
    g = S.struct(S.GatedHeads, ldo=k, ldg=k, heads=heads, head_dim=dim, norm_all=norm or 0, eps=eps, kind=kind, **t)
    p, y = weight(n, k, k), torch.zeros(1, n, device=DEV)
    sop.matvec(S.PRO_GATED, S.struct(S.Matvec, w=p.w, y=y, gated=g, n=n, k=k))
    want = p.w.cpu().double().numpy() @ v
    assert np.linalg.norm(y.cpu().double().numpy()[0] - want) < 1e-5 * np.linalg.norm(want)
