"""Jobs large enough for the bucket order: the server takes its scratch from
the library's pool only where the memory budget holds it beside the slots'
buffers, and answers the same either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,batch", [("basic", 1 << 22), ("grouped", 1 << 22), ("learned", 1 << 22)])
@pytest.mark.parametrize("room", [0, 1])
def test_scratch_within_the_budget(bt, cuda, mode, batch, room):
    import torch
    n = 1 << 24
    keys = torch.arange(0, 3 * n, 3, device=cuda, dtype=torch.int64)
    q = np.random.default_rng(batch).integers(0, 3 * n, size=batch, dtype=np.uint64)
    want = np.where(q % 3 == 0, q // 3, np.uint64(2**64 - 1))
    with bt.Tree.build(keys, torch.arange(n, device=cuda)) as t:
        if mode == "learned":
            t.learned_train(max_error=512, iterations=10)
        buffers = batch * 16 + 512
        scratch = batch * 20 + (1 << 20)
        with bt.Server(t, mode=mode, slots=1, max_batch=batch,
                       memory_budget_bytes=buffers + room * scratch) as srv:
            assert srv.stats()["slots"] == 1
            before = bt.lib().bt_workspace_allocations()
            tk, out = srv.submit(q)
            srv.wait(tk)
            assert (bt.lib().bt_workspace_allocations() > before) == bool(room)
            assert np.array_equal(out, want)
