"""Decode steps of latent attention behind a prompt: windows that fill a part of every split, more query elements and latent ranks than a
lane holds."""
import pytest
import torch

from hf2q_b200 import seqops as S
from hf2q_b200.mixers import LatentAttention
from oracle import runopel_forward as F
from tests import runopel_util as U
from tests.test_gpu_runopel_ops import mixer_of, rel, run_mixer

pytestmark = pytest.mark.gpu
DEV = "cuda"


# (heads, dim, rot, vdim, rank, window), tokens
@pytest.mark.parametrize("shape,T", [((16, 128, 64, 128, 512, 1200), 6), ((16, 128, 64, 128, 512, 1200), 540), ((16, 128, 64, 128, 512, 1200), 1300), ((3, 129, 16, 33, 513, 90), 120),
                                     ((2, 136, 8, 40, 1024, 300), 301), ((20, 512, 32, 8, 264, 130), 4), ((1, 8, 2, 31, 8, 20), 30)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_steps_behind_a_prompt(gpu_ctx, shape, T, dt):
    heads, dim, rot, vdim, rank, window = shape
    c = U.latent(heads, dim, rot, vdim, rank, window, (dim + rot) ** -0.5, 1e4)["mixer"]
    m, w, pool = mixer_of(S.SeqOps(gpu_ctx), LatentAttention, c, dt, portion=2048)
    h = torch.randn(T, 24, generator=torch.Generator().manual_seed(T)).to(dt).float().to(DEV)
    want = F.mixer_latent_attention(c, U.as_f64(w), "", h.cpu().double().numpy(), 1e-5)
    got = run_mixer(m.sop, m, pool, h, [T - 4] * (T > 4) + [1] * 4, dt)
    # as for whole sequences: f32 sums, or two bf16 roundings of the cached row and the probabilities
    assert rel(got[-4:], want[-4:]) < (3e-5 if dt == torch.float32 else 2.5e-2)
    gpu_ctx.check_status()
