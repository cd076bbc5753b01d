"""Shapes set for one operation: answers for every pair, what the tree
reports, and what is refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt", [np.uint32, np.uint64])
def test_shapes_per_operation(bt, orc, cuda, kt):
    import torch
    g = np.random.default_rng(3)
    keys = np.unique(g.integers(0, np.iinfo(kt).max, size=1 << 17, dtype=np.uint64)).astype(kt)
    q = keys[g.integers(0, len(keys), size=5003)]
    q[::2] += kt(1)
    hi = q + np.minimum(np.iinfo(kt).max - q, kt(1 << 20))
    dk, dq, dh = (torch.from_numpy(x).to(cuda) for x in (keys, q, hi))
    pts, cnt = orc.point_search(keys, keys, q), orc.range_count(keys, q, hi)
    with bt.Tree.build(dk, dk) as t:
        own = (t.info.lanes_per_query, t.info.rounds)
        assert own == bt.own_op_config(t.key_bytes, "point", 1 << 19)
        for a in bt.Tree.SEARCH_CONFIGS:
            t.set_op_config("range", *a)
            assert (t.info.lanes_per_query, t.info.rounds) == own
            assert np.array_equal(t.range_count(dq, dh).cpu().numpy(), cnt)
        t.set_op_config("point", 2, 1)
        assert (t.info.lanes_per_query, t.info.rounds) == (2, 1)
        assert np.array_equal(t.point_search(dq).cpu().numpy(), pts)
        for bad in (("point", 3, 1), ("range", 0, 1), ("point", 8, 0)):
            with pytest.raises(bt.BTreeError):
                t.set_op_config(*bad)
        with pytest.raises(bt.BTreeError):
            t.set_search_config(0, 0)
        assert (t.info.lanes_per_query, t.info.rounds) == (2, 1)
        t.set_op_config("point")
        assert (t.info.lanes_per_query, t.info.rounds) == own
        assert np.array_equal(t.point_search(dq).cpu().numpy(), pts)
