"""The autotuner's choice: a tree's own shape where the times tie (large batches
do not depend on the shape), the fastest one otherwise."""
import importlib

import pytest

at = importlib.import_module("b-tree-index-searching_b200.autotune")


@pytest.mark.parametrize("ms,default,want", [
    ({"8x1": 1.0, "4x1": 1.01, "2x1": 1.005}, "4x1", "4x1"),  # noise
    ({"8x1": 1.0, "4x1": 1.0, "2x1": 0.9}, "4x1", "2x1"),     # a real gain
    ({"8x1": 1.0, "4x1": 1.03}, "4x1", "8x1"),                # outside the tie
    ({"8x1": 1.0, "2x1": 0.99}, "4x1", "2x1"),                # default not tried
    ({"4x1": 1.0}, "4x1", "4x1"),
])
def test_pick(ms, default, want):
    assert at._pick(ms, default) == want


def test_defaults_are_tuned_configs():
    for pair in at.DEFAULT_CONFIGS.values():
        assert all(c in at.SEARCH_CONFIGS for c in pair)
