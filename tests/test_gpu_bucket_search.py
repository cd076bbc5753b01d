"""Point batches large enough to be searched by buckets, against the oracle:
key ranges that start high, fill 64 bits, crowd together or hold one key;
batches that are ragged, fall on few buckets or lie outside the keys; found
flags; and the same batch captured in a graph (the direct search)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NQ = 1 << 22  # the least batch the buckets take


def _keys(kind, kt, g):
    top = int(np.iinfo(kt).max)
    if kind == "uniform":
        return np.unique(g.integers(0, top, size=1 << 20, dtype=np.uint64, endpoint=True)).astype(kt)
    if kind == "high":  # all keys in a short stretch at the top, the all-ones key among them
        return np.sort(np.unique(np.uint64(top) - g.integers(0, 1 << 24, size=1 << 19, dtype=np.uint64))).astype(kt)
    if kind == "narrow":  # 64-bit separators staged as 32-bit offsets
        return (np.cumsum(g.integers(1, 200, size=1 << 20).astype(np.uint64)) + np.uint64(1 << 20)).astype(kt)
    if kind == "crowded":  # nearly all keys in the first bucket
        return np.append(np.arange(1, 1 << 19, dtype=np.uint64), np.uint64(top - 3)).astype(kt)
    if kind == "equal":  # runs of equal keys
        return np.sort(np.repeat(g.integers(0, top, size=1 << 15, dtype=np.uint64), 17)).astype(kt)
    return np.array([5], dtype=kt) if kind == "one" else np.array([0, 3, top], dtype=kt)


def _batch(kind, keys, kt, n, g):
    top = int(np.iinfo(kt).max)
    if kind == "mixed":
        q = keys[g.integers(0, len(keys), size=n)]
        q[::3] = g.integers(0, top, size=len(q[::3]), dtype=np.uint64, endpoint=True).astype(kt)
        q[:4] = [0, top, keys[0], keys[-1]]
        return q
    if kind == "hot":  # one key, and a few elsewhere
        q = np.full(n, keys[len(keys) // 2], dtype=kt)
        q[:100] = keys[g.integers(0, len(keys), size=100)]
        return q
    q = np.full(n, top, dtype=kt)  # outside
    q[::2] = 0
    return q


@pytest.mark.parametrize("kt,vt", [(np.uint32, np.uint32), (np.uint32, np.uint64),
                                   (np.uint64, np.uint32), (np.uint64, np.uint64)])
@pytest.mark.parametrize("kind", ["uniform", "high", "narrow", "crowded", "equal", "one", "three"])
@pytest.mark.parametrize("batch,n", [("mixed", NQ), ("mixed", NQ + 12345), ("hot", NQ + 1),
                                     ("outside", NQ + 31)])
def test_large_batches_equal_the_oracle(bt, orc, cuda, kt, vt, kind, batch, n):
    import torch
    g = np.random.default_rng(n + len(kind))
    keys = _keys(kind, kt, g)
    vals = g.integers(0, np.iinfo(vt).max, size=len(keys), dtype=np.uint64, endpoint=True).astype(vt)
    q = _batch(batch, keys, kt, n, g)
    dq = torch.from_numpy(q).to(cuda)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda)) as t:
        got = {m: t.point_search(dq, mode=m).cpu().numpy() for m in ("basic", "grouped")}
        v, f = t.point_search_found(dq)
    exp = orc.point_search(keys, vals, q)
    assert np.array_equal(got["basic"], exp)
    assert np.array_equal(got["grouped"], exp)
    assert np.array_equal(v.cpu().numpy(), exp)
    p = np.minimum(np.searchsorted(keys, q), len(keys) - 1)
    assert np.array_equal(f.cpu().numpy().astype(bool), keys[p] == q)


@pytest.mark.parametrize("kt", [np.uint32, np.uint64])
def test_windows_a_level_above_the_leaves(bt, cuda, kt):
    """2^24 keys over the whole 64 bits: the bottom level's window does not
    fit as 64-bit separators, so a level below the window is walked."""
    import torch
    n = 1 << 24
    g = torch.Generator(device=cuda)
    g.manual_seed(3)
    x = torch.randint(0, 1 << 62, (n,), generator=g, device=cuda)
    keys = torch.sort(x if kt == np.uint64 else x >> 31).values
    tk = keys if kt == np.uint64 else keys.to(torch.int32)
    with bt.Tree.build(tk, torch.arange(n, device=cuda)) as t:
        at = torch.randint(0, n, (NQ + 7,), generator=g, device=cuda)
        q = keys[at] + (at & 1)
        got = t.point_search(q if kt == np.uint64 else q.to(torch.int32)).view(torch.int64)
    p = torch.searchsorted(keys, q).clamp_(max=n - 1)
    assert torch.equal(got, torch.where(keys[p] == q, p, -1))


def test_capture_takes_the_direct_search(bt, cuda):
    import torch
    keys = torch.arange(0, 3 << 20, 3, device=cuda, dtype=torch.int32)
    with bt.Tree.build(keys, keys) as t:
        q = torch.arange(NQ, device=cuda, dtype=torch.int32)
        exp = t.point_search(q)
        out = torch.empty_like(exp)
        allocs = bt.lib().bt_workspace_allocations()
        gr = torch.cuda.CUDAGraph()
        with torch.cuda.graph(gr):
            t.point_search(q, out=out, stream=torch.cuda.current_stream())
        assert bt.lib().bt_workspace_allocations() == allocs
        gr.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int32), exp.view(torch.int32))


@pytest.mark.parametrize("kt,vt", [(np.uint32, np.uint32), (np.uint64, np.uint64)])
@pytest.mark.parametrize("kind", ["uniform", "high", "narrow", "crowded", "equal", "one", "three"])
@pytest.mark.parametrize("width", ["near", "far"])
def test_large_range_batches_equal_the_oracle(bt, orc, cuda, kt, vt, kind, width):
    """2^20 ranges and a few more (both bounds by buckets): narrow and wide
    ones, inverted ones, ends at the smallest and largest value."""
    import torch
    n = (1 << 20) + 77
    g = np.random.default_rng(len(kind))
    keys = _keys(kind, kt, g)
    top = int(np.iinfo(kt).max)
    lo = _batch("mixed", keys, kt, n, g)
    if width == "near":
        hi = np.minimum(lo, kt(top - 300)) + g.integers(0, 300, size=n).astype(kt)
    else:
        hi = _batch("mixed", keys, kt, n, g)
    lo[:4], hi[:4] = [0, 0, top, top], [0, top, top, 0]
    dlo, dhi = torch.from_numpy(lo).to(cuda), torch.from_numpy(hi).to(cuda)
    exp = orc.range_count(keys, lo, hi)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda),
                       torch.arange(len(keys), device=cuda).to(
                           torch.int32 if vt == np.uint32 else torch.int64)) as t:
        for mode in ("basic", "2d", "zorder"):
            assert np.array_equal(t.range_count(dlo, dhi, mode=mode).cpu().numpy(), exp), mode
        if width == "near" and exp.sum() < 1 << 27:
            c, o, ids = t.range_search(dlo, dhi)
            c, o, ids = c.cpu().numpy(), o.cpu().numpy(), ids.cpu().numpy()
            assert np.array_equal(c, exp)
            assert np.array_equal(o, np.cumsum(exp) - exp)
            first = np.searchsorted(keys, lo)  # values are ranks: each segment counts up
            assert np.array_equal(ids, (np.repeat(first - o.astype(np.int64), exp.astype(np.int64))
                                        + np.arange(len(ids))).astype(vt))
