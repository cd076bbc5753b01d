"""Tuning one operation leaves the other's shape alone, and a tie leaves the
tuned one the tree's own (a stand-in for the tree records what is set)."""
import importlib
import types

import pytest

at = importlib.import_module("b-tree-index-searching_b200.autotune")


class Tree:
    key_bytes, value_bytes = 8, 8
    info = types.SimpleNamespace(num_keys=1000)

    def __init__(self):
        self.shape = {"point": "own", "range": "own"}

    def set_search_config(self, g, i):
        self.shape = {"point": (g, i), "range": (g, i)}

    def set_op_config(self, op, g=0, i=0):
        self.shape[op] = (g, i) if (g, i) != (0, 0) else "own"

    def point_search(self, *a, **k):
        pass

    def range_count(self, *a, **k):
        pass


@pytest.mark.parametrize("mode,op", [("basic", "point"), ("grouped", "point"), ("range", "range")])
@pytest.mark.parametrize("tie", [True, False])
def test_the_other_operation_keeps_its_shape(monkeypatch, tmp_path, mode, op, tie):
    import torch
    other = {"point": "range", "range": "point"}[op]
    monkeypatch.setattr(torch.cuda, "current_stream", lambda *a: None)
    q = torch.zeros(1 << 12, dtype=torch.int64)
    cache = str(tmp_path / "tuned.json")
    for fresh in (True, False):  # timed, then from the cache
        tree = Tree()
        tree.shape[other] = (2, 1)
        monkeypatch.setattr(at, "_time", lambda fn, s, r: 1.0 if tie or tree.shape[op] != (8, 1) else 0.5)
        g, i, ms = at.tune(tree, q, mode=mode, hi=q, cache_path=cache)
        assert tree.shape[other] == (2, 1)
        if tie:
            assert tree.shape[op] == "own"
            assert (g, i) == importlib.import_module("b-tree-index-searching_b200").own_op_config(
                8, op, len(q))
        else:
            assert tree.shape[op] == (g, i) == (8, 1)
        assert len(ms) == 5


def test_own_shapes_are_supported_ones(bt):
    for kb in (4, 8):
        for op in ("point", "range"):
            for nq in (0, 1, 1 << 12, 1 << 13, 1 << 17, 1 << 21, 1 << 33):
                assert bt.own_op_config(kb, op, nq) in bt.Tree.SEARCH_CONFIGS
    for bad in ((5, 0), (4, 2), (8, -1)):
        assert bt.lib().bt_own_op_config(bad[0], bad[1], 1, None, None) == 1
