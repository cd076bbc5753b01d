"""Batches in bucket order that fall on one key, a few or one bucket, cut into
slices of every size the batch allows: trees whose buckets are read through L1
and larger ones, point, learned and range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt,vt", [(np.uint32, np.uint32), (np.uint32, np.uint64),
                                   (np.uint64, np.uint32), (np.uint64, np.uint64)])
@pytest.mark.parametrize("n", [1 << 14, 3 << 20])
@pytest.mark.parametrize("nq", [(1 << 18) + 1, (1 << 20) + 513, (1 << 23) + 1])
def test_batches_on_few_buckets(bt, orc, cuda, kt, vt, n, nq):
    import torch
    g = np.random.default_rng(nq + n)
    top = int(np.iinfo(kt).max)
    keys = np.unique(g.integers(0, top, size=n, dtype=np.uint64)).astype(kt)
    vals = g.integers(0, np.iinfo(vt).max, size=len(keys), dtype=np.uint64).astype(vt)
    at = len(keys) // 3
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda)) as t:
        t.learned_train(max_error=512, iterations=10)
        for span in (1, 40, 3000):
            q = keys[np.minimum(at + g.integers(0, span, size=nq), len(keys) - 1)]
            q[::4] += kt(1)
            q[:3] = [0, top, keys[-1]]
            dq = torch.from_numpy(q).to(cuda)
            exp = orc.point_search(keys, vals, q)
            for mode in ("basic", "learned"):
                v, f = t.point_search_found(dq, mode=mode)
                assert np.array_equal(v.cpu().numpy(), exp), mode
                p = np.minimum(np.searchsorted(keys, q), len(keys) - 1)
                assert np.array_equal(f.cpu().numpy().astype(bool), keys[p] == q), mode
            hi = np.roll(q, 1)
            lo = np.minimum(q, hi)
            hi = np.maximum(q, hi)
            got = t.range_count(torch.from_numpy(lo).to(cuda), torch.from_numpy(hi).to(cuda))
            assert np.array_equal(got.cpu().numpy().astype(np.int64),
                                  np.searchsorted(keys, hi, "right") - np.searchsorted(keys, lo))
