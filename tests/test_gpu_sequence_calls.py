"""What a program may do around the calls that continue a sequence, which return before the device has finished."""
import pytest
import torch

from tests import fomatar_util as U
from tests.test_gpu_fomatar import load

pytestmark = pytest.mark.gpu
LONG = 1 << 28                                           # clocks: more than a tenth of a second


def test_pinned_ids_may_be_overwritten_after_the_call(gpu_ctx):
    m, cfg, _ = load(gpu_ctx, "a", torch.float32)
    ids = torch.tensor(U.tokens(cfg, 40), dtype=torch.int32)
    slot = m.open_slot()
    want = m.extend(slot, ids, range(40))
    m.close_slot(slot)
    slot, pinned = m.open_slot(), ids.clone().pin_memory()
    torch.cuda.synchronize()
    torch.cuda._sleep(LONG)                              # the device reaches the copy of the ids long after the host has left the call
    got = m.extend(slot, pinned, range(40))
    pinned.fill_(0)
    assert torch.equal(got, want)
