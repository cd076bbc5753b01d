"""Sorted hit IDs at the edges of the sort's tiers (registers by the filling
warp, registers by a pass of its own, shared memory, global memory), with more
medium segments than the list holds, and through an allocation function that
gives nothing."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [0, 1, 2, 31, 32, 33, 64, 65, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025,
         4095, 4096, 4097, 9000, 16384, 16385, 32768, 32769]


def _tree(bt, cuda, kt, vt, n, g):
    import torch
    keys = (np.arange(n, dtype=np.uint64) * np.uint64(3) + np.uint64(1)).astype(kt)
    vals = g.permutation(n).astype(vt)
    return keys, vals, bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.from_numpy(vals).to(cuda))


def _check(t, keys, vals, first, width, cuda):
    import torch
    lo = keys[first]
    hi = keys[np.maximum(first + width - 1, 0)]
    hi = np.where(width == 0, lo - 1, hi).astype(keys.dtype)
    c, o, ids = t.range_search(torch.from_numpy(lo).to(cuda), torch.from_numpy(hi).to(cuda))
    c, o, ids = c.cpu().numpy().astype(np.int64), o.cpu().numpy().astype(np.int64), ids.cpu().numpy()
    assert np.array_equal(c, width)
    assert np.array_equal(o, np.cumsum(width) - width)
    seg = np.repeat(np.arange(len(width)), width)
    at = np.repeat(first - o, width) + np.arange(len(ids))
    want = vals[at].astype(np.uint64)
    want = want[np.lexsort((want, seg))]
    assert np.array_equal(ids.astype(np.uint64), want)


@pytest.mark.parametrize("kt,vt", [(np.uint32, np.uint32), (np.uint32, np.uint64),
                                   (np.uint64, np.uint32), (np.uint64, np.uint64)])
@pytest.mark.parametrize("top", [32, 256, 1024, 4096, 9000, 32769])
def test_segments_at_the_tiers_edges(bt, cuda, kt, vt, top):
    g = np.random.default_rng(top)
    keys, vals, t = _tree(bt, cuda, kt, vt, 80021, g)
    with t:
        width = g.permutation(np.repeat([w for w in EDGES if w <= top], 7)).astype(np.int64)
        _check(t, keys, vals, g.integers(1, 40000, size=len(width)), width, cuda)


def test_more_medium_segments_than_the_list_holds(bt, cuda):
    g = np.random.default_rng(1)
    keys, vals, t = _tree(bt, cuda, np.uint32, np.uint32, 30011, g)
    with t:
        width = np.full(66000, 300, dtype=np.int64)
        width[::1000] = 1100
        _check(t, keys, vals, g.integers(1, 28000, size=len(width)), width, cuda)


def test_allocation_that_gives_nothing(bt, cuda):
    import torch
    g = np.random.default_rng(2)
    keys, _, t = _tree(bt, cuda, np.uint32, np.uint32, 1000, g)
    refuse = ctypes.CFUNCTYPE(ctypes.c_void_p, ctypes.py_object, ctypes.c_uint64)(lambda ctx, n: None)
    with t:
        k = torch.from_numpy(keys).to(cuda)
        c, o = (torch.zeros(1000, dtype=torch.uint64, device=cuda) for _ in range(2))
        total = ctypes.c_uint64(0)
        P = ctypes.c_void_p
        st = bt.lib().bt_range_search_alloc(t.handle, 0, P(k.data_ptr()), P(k.data_ptr()), 1000,
                                            P(c.data_ptr()), P(o.data_ptr()), refuse, None,
                                            ctypes.byref(total), None)
        assert st == 3 and total.value == 1000
        assert np.array_equal(c.cpu().numpy(), np.ones(1000, dtype=np.uint64))
        assert bt.lib().bt_range_search_alloc(t.handle, 0, P(k.data_ptr()), P(k.data_ptr()), 1000,
                                              P(c.data_ptr()), P(o.data_ptr()), None, None,
                                              ctypes.byref(total), None) == 1
