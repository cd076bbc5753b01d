"""The device partition where its cut changes (one tile, one row of a warp,
the table summed by the scatter or by its own kernel, several tiles to a
chunk) and where the sort skips passes (bytes that are the same in every
key), against numpy's stable sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 1024-item tiles up to 64 rows, one short tile per CTA, whole tiles of 8192
# or 4096 items on 296 CTAs and one more
SIZES = [1023, 1025, 64 * 1024, 64 * 1024 + 1, 296 * 1024 + 33, 296 * 4096 + 1, 296 * 8192 + 1]


def _keys(kind, kt, n, g):
    bits = 8 * np.dtype(kt).itemsize
    if kind == "random":
        return g.integers(0, 1 << bits, size=n, dtype=np.uint64, endpoint=False).astype(kt)
    if kind == "equal":  # only the first pass runs
        return np.full(n, 0xA5 << (bits - 8), dtype=kt)
    if kind == "middle":  # one byte varies, not the lowest
        return (g.integers(0, 256, size=n, dtype=np.uint64) << np.uint64(8)).astype(kt) | kt(7)
    return (g.integers(0, 3, size=n, dtype=np.uint64) << np.uint64(bits - 9)).astype(kt)  # two bytes


@pytest.mark.parametrize("kt,vt", [(np.uint32, np.uint32), (np.uint64, np.uint64),
                                   (np.uint64, np.uint32)])
@pytest.mark.parametrize("kind", ["random", "equal", "middle", "top"])
@pytest.mark.parametrize("n", SIZES)
def test_sort_at_the_cuts_edges(bt, cuda, kt, vt, kind, n):
    import torch
    g = np.random.default_rng(n)
    keys = _keys(kind, kt, n, g)
    vals = np.arange(n, dtype=vt)
    k, v = bt.sort_pairs(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda))
    o = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy(), keys[o])
    assert np.array_equal(v.cpu().numpy(), vals[o])


@pytest.mark.parametrize("kt", [np.uint32, np.uint64])
@pytest.mark.parametrize("n", SIZES)
def test_group_is_stable_by_the_top_bits(bt, cuda, kt, n):
    import torch
    g = np.random.default_rng(n)
    bits = 8 * np.dtype(kt).itemsize
    keys = np.arange(1, 1001, dtype=kt) * kt(3 << (bits - 14))
    q = g.integers(0, int(keys[-1]) + 5, size=n, dtype=np.uint64).astype(kt)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda),
                       torch.arange(1000, dtype=torch.int32, device=cuda)) as t:
        grouped, perm = t.group(torch.from_numpy(q).to(cuda))
    top = np.minimum(q >> kt(int(keys[-1]).bit_length() - 8), kt(255))
    o = np.argsort(top, kind="stable")
    assert np.array_equal(perm.cpu().numpy(), o.astype(np.uint32))
    assert np.array_equal(grouped.cpu().numpy(), q[o])
