"""Windowed attention over many query tiles on tcgen05: windows and portions around the tile sizes (128 queries, 64 keys)."""
import numpy as np
import pytest
import torch

from hf2q_b200 import seqops as S
from oracle import fomatar_forward as F
from tests.test_gpu_seqops import rel, run_window

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,d,dv,window,bias", [(2, 1, 72, 128, 1, True), (3, 3, 128, 100, 63, False), (4, 2, 96, 65, 128, True), (2, 2, 128, 128, 129, False),
                                                  (1, 1, 127, 9, 300, True), (8, 2, 65, 120, 2000, False)])
def test_many_tiles(gpu_ctx, H, G, d, dv, window, bias):
    rng, T = np.random.default_rng(d + window), 643
    q, k, v = 2 * rng.standard_normal((T, H, d)), rng.standard_normal((T, G, d)), rng.standard_normal((T, G, dv))
    r1, r2 = (rng.random(H) + 0.2, rng.random(H) * 0.3) if bias else (None, None)
    to = lambda x: torch.tensor(x).to(torch.bfloat16).double().numpy()
    q, k, v = to(q), to(k), to(v)
    want = F.window_attention(q, k, v, window, d ** -0.5, r1 if bias else np.zeros(H), r2 if bias else np.zeros(H)).reshape(T, -1)
    for cuts in ([T], [127, 128, 129, 2, 257], [385, 258]):
        got = run_window(S.SeqOps(gpu_ctx), q, k, v, window, d ** -0.5, r1, r2, torch.bfloat16, cuts)
        gpu_ctx.check_status()
        assert rel(got, want) < 2 ** -8, cuts            # probabilities rounded to bf16 (2^-9 each), and their sum not


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("which", ["k", "v"])
@pytest.mark.parametrize("d,dv,window,at", [(72, 128, 500, 70), (128, 65, 100, 200), (96, 121, 128, 255), (128, 128, 1, 127)])
def test_hidden_keys_do_not_reach_a_row(gpu_ctx, bad, which, d, dv, window, at):
    """A key or value that is not finite shows in the queries that see it and in no other of the tile, before it or past its window."""
    rng, T, H = np.random.default_rng(d + window), 300, 2
    to = lambda x: torch.tensor(x).to(torch.bfloat16).double().numpy()
    q, k, v = (to(rng.standard_normal((T, H, n))) for n in (d, d, dv))
    r1, r2 = rng.random(H) + 0.2, rng.random(H) * 0.3
    want = F.window_attention(q, k, v, window, d ** -0.5, r1, r2).reshape(T, -1)
    {"k": k, "v": v}[which][at, :, 5] = bad
    blind = np.ones(T, bool)
    blind[at:at + window] = False
    got = run_window(S.SeqOps(gpu_ctx), q, k, v, window, d ** -0.5, r1, r2, torch.bfloat16, [T])
    gpu_ctx.check_status()
    assert rel(got[torch.tensor(blind)], want[blind]) < 2 ** -8
    if which == "v":
        assert not got[at:min(at + window, T)].view(-1, H, dv)[:, :, 5].isfinite().any()
