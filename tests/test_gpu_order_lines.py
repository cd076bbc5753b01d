"""Batches on either side of the sizes from which they are ordered: whether the
library takes scratch for them (it does for the order alone), and the answers,
the same on both sides.  u32 batches of the larger sizes over the key sets that
the bucket order has trouble with."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

POINT = [  # key type, keys, first ordered batch (None: never)
    (np.uint32, 1 << 16, None), (np.uint32, 1 << 20, 1 << 23), (np.uint32, 3 << 22, 1 << 22),
    (np.uint64, 1 << 16, None), (np.uint64, 1 << 18, 1 << 22),
    # a few leaf blocks: 8, 9, 64, 65, 128 and 129 of u64 keys, 16 of u32 keys
    (np.uint64, 32, None), (np.uint64, 33, 1 << 21), (np.uint64, 256, 1 << 21), (np.uint64, 257, 1 << 22),
    (np.uint64, 512, 1 << 22), (np.uint64, 513, None),
    (np.uint32, 128, None)]


def _tree(bt, torch, cuda, kt, n):
    it = torch.int32 if kt == np.uint32 else torch.int64
    keys = torch.arange(0, 3 * n, 3, device=cuda, dtype=it)
    return bt.Tree.build(keys, torch.arange(n, device=cuda, dtype=it)), it


def _allocs(bt, fn):
    before = bt.lib().bt_workspace_allocations()
    got = fn()
    return got, bt.lib().bt_workspace_allocations() - before


@pytest.mark.parametrize("kt,n,line", POINT)
@pytest.mark.parametrize("mode", ["basic", "grouped"])
def test_point_lines(bt, cuda, kt, n, line, mode):
    import torch
    t, it = _tree(bt, torch, cuda, kt, n)
    with t:
        for nq in ((1 << 24,) if line is None else (line - 1, line)):
            q = torch.randint(0, 3 * n, (nq,), device=cuda, dtype=it)
            got, allocs = _allocs(bt, lambda: t.point_search(q, mode=mode))
            assert (allocs > 0) == (line is not None and nq >= line)
            assert torch.equal(got.view(it), torch.where(q % 3 == 0, q // 3, -1).to(it))


@pytest.mark.parametrize("kt,n,line", [(np.uint32, 1 << 20, 1 << 22), (np.uint64, 1 << 20, 3 << 19),
                                       (np.uint32, 3, 1 << 20), (np.uint32, 1024, 1 << 20),
                                       (np.uint32, 1025, 1 << 22), (np.uint64, 512, 1 << 20),
                                       (np.uint64, 513, 3 << 19)])
@pytest.mark.parametrize("mode", ["basic", "2d", "zorder"])
def test_range_lines(bt, cuda, kt, n, line, mode):
    import torch
    t, it = _tree(bt, torch, cuda, kt, n)
    with t:
        for nr in (line - 1, line):
            lo = torch.randint(0, 3 * n, (nr,), device=cuda, dtype=it)
            got, allocs = _allocs(bt, lambda: t.range_count(lo, lo + 29, mode=mode))
            assert (allocs > 0) == (nr >= line)
            want = torch.clamp((lo + 32) // 3, max=n) - torch.clamp((lo + 2) // 3, max=n)
            assert torch.equal(got.view(torch.int64), want.to(torch.int64))


@pytest.mark.parametrize("gap,max_error,line", [("even", 2, 1 << 21), ("random", 4, 1 << 21),
                                                ("random", 20, 1 << 20), ("random", 80, 1 << 19),
                                                ("random", 400, 1 << 18)])
def test_learned_lines(bt, cuda, gap, max_error, line):
    import torch
    n = 1 << 19
    g = torch.Generator(device=cuda)
    g.manual_seed(max_error)
    gaps = torch.full((n,), 600, device=cuda)
    if gap == "random":
        gaps = torch.empty(n, dtype=torch.float64, device=cuda).normal_(4, 2, generator=g).exp().long() + 1
    keys = torch.cumsum(gaps, 0)
    with bt.Tree.build(keys, torch.arange(n, device=cuda)) as t:
        t.learned_train(max_error=max_error, iterations=10)
        for nq in (line - 1, line):
            at = torch.randint(0, n, (nq,), generator=g, device=cuda)
            q = keys[at] + at % 2
            got, allocs = _allocs(bt, lambda: t.point_search(q, mode="learned"))
            assert (allocs > 0) == (nq >= line)
            p = torch.searchsorted(keys, q).clamp_(max=n - 1)
            assert torch.equal(got.view(torch.int64), torch.where(keys[p] == q, p, -1))


@pytest.mark.parametrize("vt", [np.uint32, np.uint64])
@pytest.mark.parametrize("kind", ["uniform", "high", "crowded", "equal"])
def test_u32_batches_equal_the_oracle(bt, orc, cuda, vt, kind):
    import torch
    g = np.random.default_rng(len(kind))
    top = (1 << 32) - 1
    keys = {"uniform": lambda: np.unique(g.integers(0, top, size=1 << 20, endpoint=True)),
            "high": lambda: np.unique(top - g.integers(0, 1 << 24, size=1 << 19)),
            "crowded": lambda: np.append(np.arange(1, 1 << 19), top - 3),
            "equal": lambda: np.sort(np.repeat(g.integers(0, top, size=1 << 15), 17))}[kind]()
    keys = keys.astype(np.uint32)
    vals = g.integers(0, np.iinfo(vt).max, size=len(keys), dtype=np.uint64).astype(vt)
    q = keys[g.integers(0, len(keys), size=(1 << 23) + 12345)]
    q[::3] = g.integers(0, top, size=len(q[::3]), endpoint=True)
    q[:4] = [0, top, keys[0], keys[-1]]
    dq = torch.from_numpy(q).to(cuda)
    hi = q[:(1 << 22) + 77] + np.minimum(top - q[:(1 << 22) + 77], 300).astype(np.uint32)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda)) as t:
        v, f = t.point_search_found(dq)
        cnt = t.range_count(dq[:len(hi)], torch.from_numpy(hi).to(cuda)).cpu().numpy()
    assert np.array_equal(v.cpu().numpy(), orc.point_search(keys, vals, q))
    p = np.minimum(np.searchsorted(keys, q), len(keys) - 1)
    assert np.array_equal(f.cpu().numpy().astype(bool), keys[p] == q)
    assert np.array_equal(cnt, orc.range_count(keys, q[:len(hi)], hi))
