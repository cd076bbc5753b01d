"""Learned search of batches large enough for the bucket order, against the
plain search of the same batch: key widths, duplicates, keys past the largest
and below the smallest, few and many segments, buckets whose segments do not
fit in shared memory, trees of one unit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _keys(kind, kt, g):
    top = int(np.iinfo(kt).max)
    if kind == "lognormal":
        return np.cumsum(np.floor(g.lognormal(4.0, 2.0, size=1 << 20)).astype(np.uint64) + 1).astype(kt)
    if kind == "uniform":
        return np.unique(g.integers(0, top, size=1 << 20, dtype=np.uint64, endpoint=True)).astype(kt)
    if kind == "equal":
        return np.sort(np.repeat(g.integers(1, top, size=1 << 14, dtype=np.uint64), 33)).astype(kt)
    if kind == "few":
        return np.array([3, 7, 7, top], dtype=kt)
    # all keys in a short stretch at the top: one bucket per few keys
    return np.sort(np.uint64(top) - np.unique(g.integers(0, 1 << 20, size=1 << 18)).astype(np.uint64)).astype(kt)


@pytest.mark.parametrize("kt,vt", [(np.uint64, np.uint64), (np.uint64, np.uint32),
                                   (np.uint32, np.uint64), (np.uint32, np.uint32)])
@pytest.mark.parametrize("kind", ["lognormal", "uniform", "equal", "few", "top"])
@pytest.mark.parametrize("n", [1 << 18, (1 << 22) + 4567])
@pytest.mark.parametrize("target", [{"num_segments": 4096}, {"max_error": 3}, {"max_error": 100000}])
def test_learned_batches_equal_the_plain_search(bt, orc, cuda, kt, vt, kind, target, n):
    import torch
    g = np.random.default_rng(len(kind))
    keys = _keys(kind, kt, g)
    vals = g.integers(0, np.iinfo(vt).max, size=len(keys), dtype=np.uint64).astype(vt)
    top = int(np.iinfo(kt).max)
    q = keys[g.integers(0, len(keys), size=n)]
    q[::3] = g.integers(0, top, size=len(q[::3]), dtype=np.uint64, endpoint=True).astype(kt)
    q[1::7] = q[1::7] + kt(1)
    q[:6] = [0, top, keys[0], keys[-1], (int(keys[0]) - 1) % (top + 1), (int(keys[-1]) + 1) % (top + 1)]
    exp = orc.point_search(keys, vals, q)
    dq = torch.from_numpy(q).to(cuda)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda)) as t:
        try:
            t.learned_train(iterations=20, **target)
        except bt.BTreeError as e:
            assert e.name == "BT_ERR_NOT_SUPPORTED"  # more segments than the index holds
            pytest.skip("too many segments")
        assert np.array_equal(t.point_search(dq, mode="learned").cpu().numpy(), exp)
        fallback = t.learned_last_stats()[1]
        # as many full descents as the small-batch kernel at most: none, but for
        # runs of equal keys that share a threshold bucket (more than eight
        # units to walk)
        small = 0
        for part in dq.view({4: torch.int32, 8: torch.int64}[t.key_bytes]).split(1 << 17):
            t.point_search(part, mode="learned")
            small += t.learned_last_stats()[1]
        assert fallback <= small
        assert small == 0 or kind == "equal"
        v, f = t.point_search_found(dq, mode="learned")
        assert np.array_equal(v.cpu().numpy(), exp)
        p = np.minimum(np.searchsorted(keys, q), len(keys) - 1)
        assert np.array_equal(f.cpu().numpy().astype(bool), keys[p] == q)
