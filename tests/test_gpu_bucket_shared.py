"""The bucket order's scratch: two host threads with a stream each, and a
device without room for it (the direct search answers)."""
import os
import subprocess
import sys
import threading

import pytest

pytestmark = pytest.mark.gpu

N = 1 << 24

FULL = """
import importlib, torch
bt = importlib.import_module("b-tree-index-searching_b200")
n, m = 1 << 24, 1 << 24
t = bt.Tree.build(torch.arange(0, 3 * n, 3, device="cuda"), torch.arange(n, device="cuda"))
t.learned_train(max_error=512, iterations=10)
q = torch.randint(0, 3 * n, (m,), device="cuda")
want = torch.where(q % 3 == 0, q // 3, -1)
hi, out, cnt = q + 29, torch.empty_like(q), torch.empty_like(q)
wc = torch.clamp((hi + 3) // 3, max=n) - torch.clamp((q + 2) // 3, max=n)
for k in (1 << 12, 1 << 22):  # every kernel is loaded before the memory is gone
    for mode in ("basic", "learned"):
        t.point_search(q[:k], out=out, mode=mode)
    t.range_count(q[:k], hi[:k], out=cnt)
torch.equal(out, want), torch.equal(cnt, wc)
torch.cuda.synchronize()
torch.cuda.empty_cache()
rest = torch.empty(torch.cuda.mem_get_info()[0] - (128 << 20), dtype=torch.uint8, device="cuda")
for mode in ("basic", "learned", "basic"):
    out.zero_()
    t.point_search(q, out=out, mode=mode)
    assert bool((out == want).all()), mode
t.range_count(q, hi, out=cnt)
assert bool((cnt == wc).all())
del rest
torch.cuda.empty_cache()
before = bt.lib().bt_workspace_allocations()
t.point_search(q, out=out)
assert bool((out == want).all()) and bt.lib().bt_workspace_allocations() == before + 1
print("done")
"""


@pytest.mark.parametrize("mode", ["basic", "learned"])
def test_two_threads_with_a_stream_each(bt, cuda, mode):
    import torch
    keys = torch.arange(0, 3 * N, 3, device=cuda)
    errors = []
    with bt.Tree.build(keys, torch.arange(N, device=cuda)) as t:
        t.learned_train(max_error=512, iterations=10)
        torch.cuda.synchronize()

        def work(seed):
            try:
                s = torch.cuda.Stream()
                g = torch.Generator(device=cuda)
                g.manual_seed(seed)
                with torch.cuda.stream(s):
                    for k in range(8):
                        m = (1 << 22) + 1000 * seed + k
                        q = torch.randint(0, 3 * N, (m,), generator=g, device=cuda)
                        got = t.point_search(q, mode=mode, stream=s).view(torch.int64)
                        cnt = t.range_count(q, q + 29, stream=s).view(torch.int64)
                        want = torch.where(q % 3 == 0, q // 3, -1)
                        wc = torch.clamp((q + 32) // 3, max=N) - torch.clamp((q + 2) // 3, max=N)
                        s.synchronize()
                        assert torch.equal(got, want) and torch.equal(cnt, wc)
            except BaseException as e:  # noqa: B036 - reported by the test's thread
                errors.append(e)

        threads = [threading.Thread(target=work, args=(i,)) for i in (1, 2)]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
    assert not errors, errors


def test_no_room_for_the_scratch(bt, cuda):
    root = os.path.dirname(os.path.dirname(os.path.abspath(bt.__file__)))
    r = subprocess.run([sys.executable, "-c", FULL], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stderr
