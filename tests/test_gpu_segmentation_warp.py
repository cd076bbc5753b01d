"""The warp-wide segmentation against the oracle's serial restatement: chunks
of either number type (key spans around 2^31, 64-bit keys over the whole
range), runs of equal keys, hulls that reach their cap, ragged chunk ends."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNK = 1 << 14
HULL_CAP = 32


def _keys(kind, n):
    g = np.random.default_rng(n)
    if kind == "narrow":  # chunk spans far below 2^31
        return np.cumsum(g.integers(1, 4000, size=n).astype(np.uint64))
    if kind == "edge":  # chunk spans on both sides of 2^31
        return np.cumsum(g.integers(1, 262145, size=n).astype(np.uint64))
    if kind == "wide":  # the whole 64-bit range
        return np.sort(g.integers(0, 1 << 64, size=n, dtype=np.uint64, endpoint=False))
    if kind == "equal":  # runs of equal keys
        return np.sort(np.repeat(g.integers(0, 1 << 44, size=n // 20 + 1, dtype=np.uint64),
                                 20)[:n])
    i = np.arange(n, dtype=np.uint64)  # convex and concave stretches: hulls reach the cap
    k = (i % np.uint64(512)).astype(np.uint64)
    step = np.where((i // np.uint64(512)) % 2 == 0, k * k, (np.uint64(511) - k) ** 2) + np.uint64(1)
    return np.cumsum(step)


@pytest.mark.parametrize("kind", ["narrow", "edge", "wide", "equal", "bent"])
@pytest.mark.parametrize("n,eps", [(3 * CHUNK + 1, 8), (2 * CHUNK - 31, 64), (CHUNK + 2, 1 << 10),
                                   (CHUNK, (1 << 29) + 1), (33, 8)])
def test_segment_count_equals_the_oracles(bt, orc, cuda, kind, n, eps):
    import torch
    keys = _keys(kind, n)
    exp = orc.pla_segments(keys, eps, chunk=CHUNK, hull_cap=HULL_CAP, lines=False)
    dk = torch.from_numpy(keys).to(cuda)
    dv = torch.arange(n, dtype=torch.int64, device=cuda)
    with bt.Tree.build(dk, dv) as t:
        rep = t.learned_train(max_error=eps, iterations=1)
        assert rep["num_segments"] == exp
        q = torch.from_numpy(keys[:: max(1, n // 5000)].copy()).to(cuda)
        got = t.point_search_learned(q)
        assert torch.equal(got.view(torch.int64), t.point_search(q).view(torch.int64))
        assert t.learned_last_stats()[1] == 0


@pytest.mark.parametrize("kind,segments", [("narrow", 300), ("narrow", 5000), ("narrow", 70000),
                                           ("bent", 20000), ("equal", 60000), ("wide", 3000)])
def test_target_gives_the_least_bound_of_a_large_tree(bt, orc, cuda, kind, segments):
    """256 chunks and more: the bound is guessed from a sample of them, then
    counted in full on both sides."""
    import torch
    n = 257 * CHUNK + 5
    keys = _keys(kind, n)
    with bt.Tree.build(torch.from_numpy(keys).to(cuda), torch.arange(n, device=cuda)) as t:
        if kind == "bent":  # the hull cap alone cuts more segments, whatever the bound
            with pytest.raises(bt.BTreeError) as e:
                t.learned_train(num_segments=segments, iterations=1)
            assert e.value.name == "BT_ERR_NOT_SUPPORTED"
            return
        rep = t.learned_train(num_segments=segments, iterations=1)
    eps = rep["max_error"]
    count = lambda e: orc.pla_segments(keys, e, chunk=CHUNK, hull_cap=HULL_CAP, lines=False)  # noqa: E731
    assert rep["num_segments"] == count(eps) <= segments
    assert eps == 1 or count(eps - 1) > segments
