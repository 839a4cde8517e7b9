"""Prompts of the quantized decoder through panels and through f32 activations: the same bits in the logits and in the key-value cache, also
where a prompt's last portion is too short for panels, and with buffers that later prompts outgrow."""
import pytest
import torch

from hf2q_b200 import decoder as D
from tests.test_gpu_decoder import CFG, build_model

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def weights(gpu_ctx):
    return build_model(gpu_ctx, CFG)[0]


@pytest.mark.parametrize("chunk", [32, 200])
def test_same_bits(gpu_ctx, weights, chunk):
    panels, plain = (D.LlamaDecoder(gpu_ctx, CFG, weights, prefill_chunk=chunk) for _ in range(2))
    assert panels.panel_prefill
    plain.panel_prefill = False
    # portions of 9 and more, of 8 and fewer, and both, shorter and longer than the ones before; then a second part behind a first
    for parts in ([9], [8], [3], [33], [40], [41], [12], [65, 1, 20], [150], [8, 9, 100], [230]):
        ids = torch.randint(0, CFG.vocab, (sum(parts),), generator=torch.Generator().manual_seed(len(parts) * 1000 + parts[0]), dtype=torch.int32).cuda()
        got = []
        for d in (panels, plain):
            for buf in d.kv_bufs:
                for t in buf:
                    t.zero_()
            out, at = [], 0
            slot = d.open_slot()
            for n in parts:
                out += [d.extend(slot, ids[at:at + n], range(n)), d.logits.clone(), d.tok.clone()]
                at += n
            d.close_slot(slot)
            got.append(out + [t.clone() for buf in d.kv_bufs for t in buf])
        assert all(torch.equal(a, b) for a, b in zip(*got)), parts
    gpu_ctx.check_status()
