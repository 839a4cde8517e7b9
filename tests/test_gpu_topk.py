"""Choice of experts: counts around the registers' steps, ties, NaN and rows without a finite value, against the oracle."""
import numpy as np
import pytest
import torch

import hf2q_b200 as hq
import oracle
from hf2q_b200 import seqops as S

pytestmark = pytest.mark.gpu


def _rows(experts, seed):
    x = np.random.default_rng(seed).standard_normal((9, experts)).astype(np.float32)
    x[1] = 1.0                                                    # all tied: the lowest ids in order
    x[2, ::2] = np.nan
    x[3] = -np.inf
    x[4] = np.round(x[4])
    x[5, -1] = 80.0                                               # all others vanish
    return x


@pytest.mark.parametrize("experts", [1, 2, 31, 32, 33, 64, 65, 128, 129, 256, 257, 1000])
def test_softmax_choice(gpu_ctx, experts):
    x = _rows(experts, experts)
    for k in {1, min(8, experts), min(40, experts)}:
        ids, w = hq.moe_softmax_topk(gpu_ctx, torch.from_numpy(x).cuda(), k)
        want_ids, want_w = oracle.softmax_topk_renorm(x, k)
        assert np.array_equal(ids.cpu().numpy().astype(np.int64), want_ids.astype(np.int64))
        np.testing.assert_allclose(w.cpu().numpy(), want_w, rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("experts", [3, 32, 200, 300])
def test_sigmoid_choice(gpu_ctx, experts):
    x, k = _rows(experts, experts + 1), min(5, experts)
    x = np.delete(x, 2, axis=0)
    xd, ids, w = torch.from_numpy(x).cuda(), torch.zeros(8, k, dtype=torch.int32, device="cuda"), torch.zeros(8, k, device="cuda")
    S.SeqOps(gpu_ctx).sigmoid_topk(xd, ids, w, 8, experts, k)
    p = 1 / (1 + np.exp(-x.astype(np.float64)))
    got = w.cpu().numpy()
    np.testing.assert_allclose(got, -np.sort(-p, axis=1)[:, :k], rtol=1e-6)
    np.testing.assert_allclose(np.take_along_axis(p, ids.cpu().numpy().astype(np.int64), 1), got, rtol=1e-6)
    assert list(ids[1].cpu().numpy()) == list(range(k))           # the tied row
