"""Learned batches in bucket order over keys that are regular but for a short
stretch, where most segments lie: the fullest bucket's part of the index is
many times the average one's, or more than the shared memory holds.  Answers
equal the oracle's and no query takes the full descent, whether the batch is
spread over the keys or falls on the stretch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _keys(n, at, crowd, kt, g):
    """n keys 600 apart, but for `crowd` of them from `at` on, whose gaps are
    lognormal with a mean of 600 / 3.3."""
    gap = np.full(n, 600, dtype=np.uint64)
    gap[at:at + crowd] = np.floor(g.lognormal(3.2, 2.0, size=crowd)).astype(np.uint64) + 1
    return np.cumsum(gap).astype(kt)


@pytest.mark.parametrize("kt,vt,n,crowd,target", [
    (np.uint64, np.uint64, 1 << 20, 1 << 15, {"num_segments": 4096}),   # 10x the average
    (np.uint64, np.uint32, 1 << 20, 1 << 15, {"max_error": 2}),
    (np.uint32, np.uint32, 1 << 20, 1 << 15, {"num_segments": 4096}),
    (np.uint64, np.uint64, 1 << 24, 1 << 18, {"max_error": 1}),         # above 200 KB a bucket
])
def test_crowded_segments_take_no_full_descent(bt, orc, cuda, kt, vt, n, crowd, target):
    import torch
    g = np.random.default_rng(n + crowd)
    at = n // 3
    keys = _keys(n, at, crowd, kt, g)
    vals = g.integers(0, np.iinfo(vt).max, size=n, dtype=np.uint64).astype(vt)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda)) as t:
        t.learned_train(iterations=20, **target)
        for span in ((0, n), (at, at + crowd)):
            q = keys[g.integers(*span, size=(1 << 22) + 77)]
            q[::5] += kt(1)
            q[:2] = [0, np.iinfo(kt).max]
            dq = torch.from_numpy(q).to(cuda)
            v, f = t.point_search_found(dq, mode="learned")
            assert t.learned_last_stats()[1] == 0
            assert np.array_equal(v.cpu().numpy(), orc.point_search(keys, vals, q))
            p = np.minimum(np.searchsorted(keys, q), n - 1)
            assert np.array_equal(f.cpu().numpy().astype(bool), keys[p] == q)


@pytest.mark.parametrize("kt", [np.uint32, np.uint64])
def test_a_run_of_the_largest_key(bt, orc, cuda, kt):
    """Many equal keys at the end: the last bucket ends at the first of them."""
    import torch
    g = np.random.default_rng(8)
    keys = np.sort(np.concatenate([np.unique(g.integers(0, 1 << 31, size=1 << 18)),
                                   np.full(5000, (1 << 31) + 9)]).astype(kt))
    vals = np.arange(len(keys)).astype(kt)
    q = keys[g.integers(0, len(keys), size=1 << 22)]
    q[::3] = keys[-1]
    q[1::9] = keys[-1] + kt(1)
    q[:2] = [0, np.iinfo(kt).max]
    exp = orc.point_search(keys, vals, q)
    dq = torch.from_numpy(q).to(cuda)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda)) as t:
        t.learned_train(max_error=16, iterations=20)
        for mode in ("basic", "learned"):
            assert np.array_equal(t.point_search(dq, mode=mode).cpu().numpy(), exp), mode
        cnt = t.range_count(dq, dq).cpu().numpy()
    assert np.array_equal(cnt, np.searchsorted(keys, q, "right") - np.searchsorted(keys, q))
