"""A tree image loaded on a stream of the caller's that does not wait for the
default one: searched at once on that stream, direct and by buckets."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1000, 1 << 22])
def test_load_on_a_side_stream(bt, cuda, tmp_path, m):
    import torch
    n = 1 << 24
    path = str(tmp_path / "tree.img")
    keys = torch.arange(0, 3 * n, 3, device=cuda, dtype=torch.int64)
    with bt.Tree.build(keys, torch.arange(n, device=cuda)) as t:
        t.save(path)
    q = torch.randint(0, 3 * n, (m,), device=cuda)
    want = torch.where(q % 3 == 0, q // 3, -1)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    h, out = ctypes.c_void_p(), torch.empty(m, dtype=torch.int64, device=cuda)
    P = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    torch.cuda.synchronize()
    L = bt.lib()
    assert L.bt_load(path.encode(), ctypes.c_void_p(s.cuda_stream), ctypes.byref(h)) == 0
    assert L.bt_point_search(h, 0, P(q), m, P(out), ctypes.c_void_p(s.cuda_stream)) == 0
    s.synchronize()
    assert torch.equal(out, want)
    assert L.bt_destroy(h) == 0
