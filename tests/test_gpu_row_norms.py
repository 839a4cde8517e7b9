"""Row prologues of portions with a row's groups in registers: few and many rows a CTA, widths that leave threads idle, padded pitches."""
import numpy as np
import pytest
import torch

from hf2q_b200 import seqops as S
from oracle import fomatar_forward as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def f32(a):
    return torch.tensor(np.asarray(a), dtype=torch.float32, device=DEV)


def rel(got, want):
    got = got.detach().cpu().double().numpy().reshape(want.shape)
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


@pytest.mark.parametrize("m,width", [(2, 4), (3, 2048), (297, 2048), (700, 4096), (1200, 1028), (5, 4100)])
@pytest.mark.parametrize("pair,shift", [(False, False), (True, False), (False, True), (True, True)])
def test_pre_norm(gpu_ctx, m, width, pair, shift):
    sop, rng, eps, ldo = S.SeqOps(gpu_ctx), np.random.default_rng(m + width), 1e-5, S.pad8(width)
    x, a, b, add0 = (rng.standard_normal((m, width)) for _ in range(4))
    an, bn, step, norm, mu, before = (rng.standard_normal(width) for _ in range(6))
    rows = x + add0 + step + (0.5 * (F.rms(a, eps) * an + F.rms(b, eps) * bn) if pair else 0.0)
    h = F.rms(rows, eps) * norm
    want = h + (np.vstack([before[None], h[:-1]]) - h) * mu if shift else h
    state, pos = f32(np.stack([before, before])), torch.tensor([3], dtype=torch.int32, device=DEV)
    x_out, out, last = torch.zeros(m, width, device=DEV), torch.full((m, ldo), 3.0, device=DEV), torch.zeros(1, width, device=DEV)
    t = dict(x=f32(x), add0=f32(add0), step=f32(step), norm=f32(norm))
    if pair:
        t |= dict(a=f32(a), b=f32(b), a_norm=f32(an), b_norm=f32(bn))
    if shift:
        t |= dict(shift=f32(mu), shift_state=state, pos=pos)
    p = S.struct(S.PreNorm, x_out=x_out, eps=eps, width=width, **t)
    sop.pre_norm(p, m, out, last if shift else None)
    assert rel(x_out, rows) < 1e-6 and rel(out[:, :width], want) < 2e-6 and float(out[:, width:].abs().sum()) == 0.0
    assert not shift or rel(last, h[-1:]) < 1e-6
    bf = torch.full((m, ldo), 3.0, dtype=torch.bfloat16, device=DEV)
    sop.pre_norm(p, m, bf, last if shift else None)
    assert torch.equal(bf, out.bfloat16())


@pytest.mark.parametrize("m,width", [(1, 8), (3, 2048), (300, 2048), (700, 4096), (1200, 1028), (5, 4100)])
@pytest.mark.parametrize("streams,x_streams,parts", [(1, 1, 1), (2, 2, 0), (4, 4, 1), (4, 1, 4), (3, 3, 5), (4, 4, 9), (5, 5, 1)])
def test_hyper_norm(gpu_ctx, m, width, streams, x_streams, parts):
    sop, rng, eps, ldo = S.SeqOps(gpu_ctx), np.random.default_rng(m + width + streams), 1e-5, S.pad8(width)
    x, c_in, norm = rng.standard_normal((m, x_streams, width)), rng.standard_normal(streams), rng.standard_normal(width)
    mix, gain, y = rng.standard_normal((streams, streams)), rng.standard_normal(streams), rng.standard_normal((m, max(parts, 1), width))
    old = np.broadcast_to(x, (m, streams, width))
    new = np.einsum("ab,maw->mbw", mix, old) + gain[:, None] * y.sum(1, keepdims=True) if parts else old
    u = np.einsum("s,msw->mw", c_in, new)
    want = F.rms(u, eps) * norm
    in_place = parts and x_streams == streams
    xg = f32(x)
    x_out = xg if in_place else torch.zeros(m, streams, width, device=DEV)
    t = dict(x=xg, c_in=f32(c_in), norm=f32(norm))
    if parts:
        t |= dict(y=f32(y), mix=f32(mix), out=f32(gain), x_out=x_out)
    p = S.struct(S.Hyper, x_streams=x_streams, streams=streams, width=width, y_parts=parts or None, eps=eps, **t)
    out = torch.full((m, ldo), 3.0, device=DEV)
    sop.hyper_norm(p, m, out)
    # the streams are mixed with weights of either sign: a few roundings of the largest term
    assert rel(out[:, :width], want) < 5e-6 and float(out[:, width:].abs().sum()) == 0.0
    assert not parts or rel(x_out, new) < 2e-6
