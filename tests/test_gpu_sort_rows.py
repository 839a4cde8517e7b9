"""Counting sort of routed rows: one CTA, a cluster's shares, and more rows than its threads hold; ids out of range are left out."""
import pytest
import torch

import hf2q_b200 as hq
from hf2q_b200 import seqops as S

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows,experts,tile", [(1, 1, 32), (37, 5, 32), (2048, 256, 128), (2049, 256, 128), (2064, 7, 64), (16384, 256, 128), (131072, 64, 128),
                                               (131089, 1500, 32)])
@pytest.mark.parametrize("bad", [False, True])
def test_sorted_order(gpu_ctx, rows, experts, tile, bad):
    g = torch.Generator(device=DEV).manual_seed(rows + experts)
    ids = torch.randint(0, experts, (rows,), generator=g, device=DEV, dtype=torch.int32)
    ids[: rows // 3] = experts // 2                               # one expert has many
    if bad:
        ids[::5] = experts + 3
    x = torch.zeros(rows, 8, dtype=torch.bfloat16, device=DEV)
    x[:, 0] = (torch.arange(rows, device=DEV) % 251).bfloat16()
    header, perm = torch.zeros(64, dtype=torch.int32, device=DEV), torch.full((rows,), -1, dtype=torch.int32, device=DEV)
    tiles, xg = torch.zeros(rows // tile + min(rows, experts) + 1, 4, dtype=torch.int32, device=DEV), torch.zeros_like(x)
    ctx = gpu_ctx
    ctx._check(ctx._lib.hf2q_cuda_sort_rows(ctx._h, ctx._stream(), ids.data_ptr(), rows, 1, experts, tile, x.data_ptr(), 2, 8, header.data_ptr(), tiles.data_ptr(),
                                            perm.data_ptr(), xg.data_ptr()))
    if bad:
        with pytest.raises(hq.Hf2qError):
            ctx.check_status()
    else:
        ctx.check_status()
    valid = torch.nonzero(ids < experts).flatten()
    counts = torch.bincount(ids[valid].long(), minlength=experts)
    n_tiles, n = int(header[0]), int(header[1])
    assert n == len(valid) and n_tiles == int(((counts + tile - 1) // tile).sum())
    order = perm[:n].long()
    assert torch.equal(order.sort().values, valid)
    assert torch.equal(ids[order].long(), torch.repeat_interleave(torch.arange(experts, device=DEV), counts))
    assert torch.equal(xg[:n], x[order])
    t = tiles[:n_tiles].long()
    first = torch.cumsum(counts, 0) - counts
    per = (counts + tile - 1) // tile
    e = torch.repeat_interleave(torch.arange(experts, device=DEV), per)
    j = torch.arange(n_tiles, device=DEV) - torch.repeat_interleave(torch.cumsum(per, 0) - per, per)
    assert torch.equal(t[:, 0], e) and torch.equal(t[:, 1], first[e] + j * tile) and torch.equal(t[:, 2], torch.minimum(counts[e] - j * tile, torch.tensor(tile, device=DEV)))
