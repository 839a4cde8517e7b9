"""One token of the recurrent mixers against f64: ranks around what a group of lanes holds, four taps in place and off 16 bytes, other counts,
every position of the ring."""
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


def f32(a, off=0):
    """On the device, `off` floats behind a 16-byte boundary."""
    a = np.asarray(a)
    t = torch.zeros(a.size + off, device=DEV)[off:].view(a.shape)
    t.copy_(torch.tensor(a, dtype=torch.float32))
    return t


def rel(got, want):
    got = got.detach().cpu().double().numpy().reshape(want.shape)
    return float(np.linalg.norm(got - want) / np.linalg.norm(want))


def silu(x):
    return x * F.sigmoid(x)


def conv(ring, w, now, pos, bias=0.0):
    taps = w.shape[1]
    return silu(bias + now * w[:, -1] + sum(ring[:, (pos - j) % taps] * w[:, taps - 1 - j] for j in range(1, taps)))


@pytest.mark.parametrize("H,G,d,dv,taps,rank,off", [(4, 2, 128, 128, 4, 128, 0), (2, 2, 128, 40, 4, 8, 0), (3, 1, 100, 33, 4, 120, 0), (2, 1, 256, 64, 4, 136, 0),
                                                    (2, 1, 32, 16, 4, 264, 0), (2, 2, 224, 7, 4, 128, 1), (2, 1, 64, 16, 5, 16, 0), (2, 1, 20, 8, 1, 24, 0)])
def test_delta(sop, H, G, d, dv, taps, rank, off):
    rng, dp = np.random.default_rng(d + rank), S.pad32(d)
    ch = 2 * G * d + H * dv
    x, beta, a1, g1 = rng.standard_normal(ch), rng.standard_normal(H), rng.standard_normal(rank), rng.standard_normal(rank)
    w, a_log, dt = rng.standard_normal((ch, taps)), rng.standard_normal(H) - 1, rng.standard_normal(H * d) - 1
    a2, g2 = (torch.tensor(rng.standard_normal((n, rank)) / rank ** 0.5).to(torch.bfloat16).to(DEV) for n in (H * d, H * dv))
    s0 = np.zeros((H, dv, dp))
    s0[:, :, :d] = rng.standard_normal((H, dv, d))
    proj = f32(np.concatenate([x, beta, a1, g1]))
    unit = lambda v: v / np.sqrt((v * v).sum(-1, keepdims=True) + 1e-6)
    for pos in range(taps):
        ring = rng.standard_normal((ch, taps))
        y = conv(ring, w, x, pos)
        q, k = (np.repeat(unit(y[i * G * d:(i + 1) * G * d].reshape(G, d)), H // G, 0) for i in range(2))
        decay = np.exp(-np.exp(a_log)[:, None] * F.softplus((a2.cpu().double().numpy() @ a1 + dt).reshape(H, d)))
        st = s0[:, :, :d] * decay[:, None]
        u = F.sigmoid(beta)[:, None] * (y[2 * G * d:].reshape(H, dv) - np.einsum("hvd,hd->hv", st, k))
        st = st + u[:, :, None] * k[:, None]
        want = np.einsum("hvd,hd->hv", st, q) * d ** -0.5
        t = dict(q_conv=f32(w[:G * d], off), k_conv=f32(w[G * d:2 * G * d], off), v_conv=f32(w[2 * G * d:], off), a_log=f32(a_log), dt_bias=f32(dt), a2=a2, g2=g2,
                 conv_state=f32(ring, off), s=f32(s0), pos=torch.tensor([pos + 3 * taps], dtype=torch.int32, device=DEV))
        a = S.struct(S.Delta, proj=proj, ld=proj.numel(), q_off=0, k_off=G * d, v_off=2 * G * d, b_off=ch, a1_off=ch + H, g1_off=ch + H + rank, heads=H, kv_heads=G, dim=d,
                     vdim=dv, taps=taps, a_rank_ld=rank, g_rank_ld=rank, **t)
        out, gate = torch.zeros(1, H * dv, device=DEV), torch.zeros(1, H * dv, device=DEV)
        sop.delta_step(a, out, gate)
        ring[:, pos] = x
        assert rel(out, want) < 5e-6 and rel(gate, g2.cpu().double().numpy() @ g1) < 2e-6
        assert rel(t["s"][:, :, :d], st) < 2e-6 and float(t["s"][:, :, d:].abs().sum()) == 0.0 and rel(t["conv_state"], ring) < 1e-7


@pytest.mark.parametrize("H,G,n,dv,taps,off", [(4, 2, 128, 64, 4, 0), (2, 1, 256, 40, 4, 0), (3, 3, 20, 7, 4, 0), (2, 2, 224, 16, 4, 1), (2, 1, 64, 16, 5, 0), (2, 1, 32, 16, 1, 0)])
def test_ssd(sop, H, G, n, dv, taps, off):
    rng, dp, inner = np.random.default_rng(n + dv), S.pad32(n), H * dv
    ch = inner + 2 * G * n
    x, dt = rng.standard_normal(ch), rng.standard_normal(H)
    w, bias, dtb, a_log, skip = rng.standard_normal((ch, taps)), rng.standard_normal(ch), rng.standard_normal(H), rng.standard_normal(H) - 1, rng.standard_normal(H)
    s0 = np.zeros((H, dv, dp))
    s0[:, :, :n] = rng.standard_normal((H, dv, n))
    proj = f32(np.concatenate([x, dt]))
    for pos in range(taps):
        ring = rng.standard_normal((ch, taps))
        y = conv(ring, w, x, pos, bias)
        v, b, c = y[:inner].reshape(H, dv), *(np.repeat(y[inner + i * G * n:inner + (i + 1) * G * n].reshape(G, n), H // G, 0) for i in range(2))
        step = F.softplus(dt + dtb)
        st = s0[:, :, :n] * np.exp(-np.exp(a_log) * step)[:, None, None] + step[:, None, None] * v[:, :, None] * b[:, None]
        want = np.einsum("hvn,hn->hv", st, c) + skip[:, None] * v
        t = dict(conv=f32(w, off), conv_bias=f32(bias), dt_bias=f32(dtb), a_log=f32(a_log), d=f32(skip), conv_state=f32(ring, off), s=f32(s0),
                 pos=torch.tensor([pos + 3 * taps], dtype=torch.int32, device=DEV))
        out = torch.zeros(1, inner, device=DEV)
        sop.ssd_step(S.struct(S.Ssd, proj=proj, ld=ch + H, off=0, heads=H, groups=G, state=n, vdim=dv, taps=taps, **t), out)
        ring[:, pos] = x
        assert rel(out, want) < 5e-6 and rel(t["s"][:, :, :n], st) < 2e-6 and rel(t["conv_state"], ring) < 1e-7
