"""Long portions run a layer's recurrence on a second stream: the same bits as in turn, from whichever stream the call comes."""
import pytest
import torch

from hf2q_b200 import mixers
from hf2q_b200.fomatar import FomatarConfig, FomatarDecoder
from tests import fomatar_util as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_same_bits_as_in_turn(gpu_ctx, dtype, monkeypatch):
    cfg = U.CONFIGS["c"]
    m = FomatarDecoder(gpu_ctx, FomatarConfig(cfg), U.weights(cfg, 0).__getitem__, dtype=dtype, max_seq=1024)
    ids = torch.tensor(U.tokens(cfg, 700, 5), dtype=torch.int32)

    def run(line):
        monkeypatch.setattr(mixers, "BESIDE_TOKENS", line)
        slot, out, at = m.open_slot(), [], 0
        for c in (256, 1, 300, 143):
            out.append(m.extend(slot, ids[at:at + c], range(c)).clone())
            at += c
        m.close_slot(slot)
        return torch.cat(out)

    want = run(1 << 30)
    for _ in range(3):
        assert torch.equal(run(2), want)
    assert torch.equal(run(256), want)
    with torch.cuda.stream(torch.cuda.Stream()):
        assert torch.equal(run(2), want)
    m.ctx.check_status()
