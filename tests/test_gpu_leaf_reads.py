"""The direct point search's two ways of reading leaf blocks (a thread per
query, a lane pair per query): trees on both sides of the size where 4-byte
keys change over, every search shape, ragged batches, the largest key value
and the keys around a block's end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 64 MiB of leaf blocks are 2^23 u32 keys with u32 values
SIZES = [1, 7, 8, 9, 1 << 12, (1 << 23) - 3, (1 << 23) + 5]


@pytest.mark.parametrize("kb,vb", [(4, 4), (4, 8), (8, 4), (8, 8)])
@pytest.mark.parametrize("n", SIZES)
def test_both_ways_equal_a_sorted_lookup(bt, cuda, kb, vb, n):
    import torch
    it = {4: torch.int32, 8: torch.int64}
    g = torch.Generator(device=cuda)
    g.manual_seed(n)
    top = (1 << 32) - 1 if kb == 4 else (1 << 62)
    keys = torch.cumsum(torch.randint(1, max(2, 2 * (top // (n + 1)) - 1), (n,), generator=g,
                                      device=cuda, dtype=torch.int64), 0)
    keys = torch.unique(keys.clamp_(max=top))  # a run above the top becomes the top itself
    n = len(keys)
    vals = torch.arange(n, device=cuda)
    at = torch.randint(0, n, (70001,), generator=g, device=cuda)
    q = keys[at] + torch.randint(0, 3, (70001,), generator=g, device=cuda) - 1
    q = torch.cat([q.clamp_(0, top), keys[:40], keys[-40:],
                   torch.tensor([0, top, int(keys[0]), int(keys[-1])], device=cuda)])
    p = torch.searchsorted(keys, q).clamp_(max=n - 1)
    hit = keys[p] == q
    want = torch.where(hit, vals[p], -1)
    with bt.Tree.build(keys.to(it[kb]), vals.to(it[vb])) as t:
        for cfg in (None,) + bt.Tree.SEARCH_CONFIGS:
            if cfg:
                t.set_search_config(*cfg)
            for m in (1, 31, 33, len(q)):
                v, f = t.point_search_found(q[-m:].to(it[kb]))
                assert torch.equal(v.view(it[vb]).to(torch.int64), want[-m:]), (cfg, m)
                assert torch.equal(f.to(torch.bool), hit[-m:]), (cfg, m)
