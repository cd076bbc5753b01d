"""The staged-window kernel of grouped batches (2^21 queries and more), reached
through the grouping step and the search of its output, and, with found flags,
by grouped batches on keys that the bucket order does not take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NQ = (1 << 21) + 77
TYPES = [(np.uint32, np.uint32), (np.uint32, np.uint64), (np.uint64, np.uint32), (np.uint64, np.uint64)]


def _batch(keys, kt, g, nq):
    hi = int(np.iinfo(kt).max)
    q = keys[g.integers(0, len(keys), size=nq)]
    q[::3] = g.integers(0, hi, size=len(q[::3]), dtype=np.uint64, endpoint=True).astype(kt)
    q[:4] = [0, 1, hi, hi - 1]
    return q


@pytest.mark.parametrize("kt,vt", TYPES)
@pytest.mark.parametrize("n", [1, 37, 200, 5000, 300001, 1 << 22])
def test_grouped_batches(bt, orc, cuda, kt, vt, n):
    import torch
    g = np.random.default_rng(n)
    if n == 200:  # single key values per group, the last group holds every larger query
        keys = np.arange(n, dtype=kt)
    else:
        keys = np.unique(g.integers(0, int(np.iinfo(kt).max), size=n, dtype=np.uint64)).astype(kt)
    vals = g.integers(0, np.iinfo(vt).max, size=len(keys), dtype=np.uint64).astype(vt)
    q = _batch(keys, kt, g, NQ)
    if n == 200:
        q = np.minimum(q, kt(300))
    dq = torch.from_numpy(q).to(cuda)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda)) as t:
        grouped, perm = t.group(dq)
        got = t.search_grouped_batch(grouped, perm).cpu().numpy()
    assert np.array_equal(got, orc.point_search(keys, vals, q))


@pytest.mark.parametrize("kt,vt", TYPES)
def test_found_flags_of_crowded_keys(bt, orc, cuda, kt, vt):
    """Nearly all keys in the first bucket: grouped batches take the groups."""
    import torch
    g = np.random.default_rng(9)
    top = int(np.iinfo(kt).max)
    keys = np.append(np.arange(1, 1 << 19, dtype=np.uint64), np.uint64(top)).astype(kt)
    vals = g.integers(0, np.iinfo(vt).max, size=len(keys), dtype=np.uint64).astype(vt)
    vals[::7] = np.iinfo(vt).max  # stored values equal to the miss marker
    q = g.integers(0, 1 << 20, size=(1 << 23) + 5, dtype=np.uint64).astype(kt)
    q[:4] = [0, top, keys[0], keys[-2]]
    dq = torch.from_numpy(q).to(cuda)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda)) as t:
        before = bt.lib().bt_workspace_allocations()
        out, found = t.point_search_found(dq, mode="grouped")
        assert bt.lib().bt_workspace_allocations() - before == 3  # the groups' two arrays and table
        out, found = out.cpu().numpy(), found.cpu().numpy()
    assert np.array_equal(out, orc.point_search(keys, vals, q))
    assert np.array_equal(found.astype(bool), np.isin(q, keys))
