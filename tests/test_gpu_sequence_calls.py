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


@pytest.mark.parametrize("design", ["fomatar", "runopel"])
def test_no_call_allocates_pinned_memory(gpu_ctx, design):
    from tests import test_gpu_runopel as R
    m, cfg, _ = load(gpu_ctx, "a", torch.float32) if design == "fomatar" else R.load(gpu_ctx, "a", torch.float32)
    ids = torch.randint(0, cfg["vocab"], (70,), dtype=torch.int32)
    torch.cuda.synchronize()
    before = torch.cuda.host_memory_stats()["num_host_alloc"]
    slot = m.open_slot()
    for a, b, want in [(0, 40, [39]), (40, 41, [0]), (41, 60, [3, 7, 18]), (60, 61, []), (61, 70, [])]:
        m.extend(slot, ids[a:b], want)
    assert torch.cuda.host_memory_stats()["num_host_alloc"] == before


def test_staging_wraps_behind_its_copies(gpu_ctx):
    from hf2q_b200.decoder import Staging
    st, sent, got = Staging(256, torch.device("cuda", 0)), [], []
    torch.cuda.synchronize()
    torch.cuda._sleep(LONG // 8)
    for i in range(1, 90):                               # sizes on both sides of the buffer's
        sent.append(torch.arange(i, dtype=torch.int64) * 1000 + i)
        got.append(st.to_device(sent[-1]))
    for a, b in zip(sent, got):
        assert torch.equal(a, b.cpu())


def test_calls_on_alternating_streams(gpu_ctx):
    """Each call works on what the last one left, although that may still be waiting on another stream."""
    from hf2q_b200.engine import Engine, Entry
    cuts, ids = [40, 1, 1, 90, 2, 1, 1], None

    def rows(streams):
        nonlocal ids
        m, cfg, _ = load(gpu_ctx, "a", torch.float32, prefill_chunk=64)          # (the larger portion grows the scratch buffers)
        ids = U.tokens(cfg, sum(cuts)) if ids is None else ids
        e, out, at = Engine(m), [], 0
        torch.cuda.synchronize()
        for i, n in enumerate(cuts):
            with torch.cuda.stream(streams[i % len(streams)]):
                torch.cuda._sleep(LONG // 4)
                out.append(e.step([Entry("r", list(ids[at:at + n]), [n - 1])]))
            at += n
        torch.cuda.synchronize()
        return torch.cat(out)

    one = rows([torch.cuda.Stream()])
    assert torch.equal(rows([torch.cuda.Stream(), torch.cuda.Stream()]), one)


@pytest.mark.parametrize("design", ["fomatar", "runopel"])
@pytest.mark.parametrize("n,want", [(2, [1]), (3, [0, 2]), (4, [1, 1, 2]), (3, [2, 2]), (1, [0])])
def test_as_many_rows_as_tokens(gpu_ctx, design, n, want):
    """The rows asked for and the last one can be as many as the portion's tokens without being those tokens."""
    from tests import test_gpu_runopel as R
    m, cfg, _ = load(gpu_ctx, "a", torch.float32, n_slots=2) if design == "fomatar" else R.load(gpu_ctx, "a", torch.float32, n_slots=2)
    ids = torch.tensor(U.tokens(cfg, n), dtype=torch.int32)
    every = m.extend(m.open_slot(), ids, range(n))
    some = m.extend(m.open_slot(), ids, want)
    assert (some - every[want]).norm() <= 1e-5 * every[want].norm()          # (other row counts take other products of the head)
