"""Host-buffer searches around the pipeline's chunk sizes: one chunk, a few on
the three slots, a slot used again, a short last chunk, every mode."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kt", [np.uint32, np.uint64])
@pytest.mark.parametrize("nq", [1, (1 << 20) - 1, 1 << 20, (1 << 20) + 1, (3 << 20) + 7, (5 << 20) - 3,
                                (1 << 23) + 9])
def test_chunked_batches(bt, cuda, kt, nq):
    import torch
    n = 1 << 21
    it = torch.int32 if kt == np.uint32 else torch.int64
    g = np.random.default_rng(nq)
    q = g.integers(0, 3 * n, size=nq, dtype=np.uint64).astype(kt)
    want = np.where(q % 3 == 0, q // 3, np.iinfo(kt).max).astype(kt)
    below = lambda x: np.minimum((x.astype(np.int64) + 2) // 3, n)  # noqa: E731
    cnt = below(q + kt(31)) - below(q)
    keys = torch.arange(0, 3 * n, 3, device=cuda, dtype=it)
    with bt.Tree.build(keys, torch.arange(n, device=cuda, dtype=it)) as t:
        t.learned_train(max_error=512, iterations=10)
        for mode in ("basic", "grouped", "learned"):
            assert np.array_equal(t.point_search(q, mode=mode), want), mode
        for mode in ("basic", "zorder"):
            assert np.array_equal(t.range_count(q, q + kt(30), mode=mode).astype(np.int64), cnt), mode
