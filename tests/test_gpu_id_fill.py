"""Hit IDs of few and of many ranges, short, at the edge of what a warp takes
alone and long, mixed and in one place of the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt,vt", [(np.uint32, np.uint32), (np.uint32, np.uint64),
                                   (np.uint64, np.uint32), (np.uint64, np.uint64)])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("nr", [1, 7, 8, 9, 257, 9473, 20001, 70003])
def test_ids_of_short_and_long_ranges(bt, cuda, kt, vt, shuffled, nr):
    import torch
    n = 1 << 20
    g = np.random.default_rng(nr)
    keys = (np.arange(n, dtype=np.uint64) * 3 + 5).astype(kt)
    vals = (g.permutation(n) if shuffled else np.arange(n)).astype(vt)
    w = g.integers(0, 60, size=nr)
    edge = [0, 1, 255, 256, 257, 2047, 2048, 2049, 2056, 4096 + 7, 16 * 2048 + 1]
    at = g.integers(0, nr, size=min(nr, 40))
    w[at] = g.choice(edge, size=len(at))
    w[nr // 2:nr // 2 + 12] = edge[-1]  # neighbours
    a = g.integers(0, n - w.max(), size=nr)
    lo = keys[a]
    hi = keys[np.maximum(a + w, 1) - 1]
    lo[w == 0], hi[w == 0] = keys[0] + kt(1), keys[0] + kt(1)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda)) as t:
        c, o, ids = (x.cpu().numpy() for x in t.range_search(torch.from_numpy(lo).to(cuda),
                                                             torch.from_numpy(hi).to(cuda)))
    assert np.array_equal(c, w)
    assert np.array_equal(o, np.cumsum(w) - w)
    seg = np.repeat(np.arange(nr), w)
    got = vals[np.arange(len(seg)) - o[seg].astype(np.int64) + a[seg]]
    if shuffled:
        got = got[np.lexsort((got, seg))]
    assert np.array_equal(ids, got)
