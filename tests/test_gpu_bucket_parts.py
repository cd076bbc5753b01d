"""Batches that the bucket order takes in several parts: answers and found flags
of every part, learned and plain, and the ranges'; and the scratch that such a
batch leaves in the library's memory pool."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

N = 1 << 24  # keys 0, 3, 6, ...: key 3 r has rank r

POOL = """
import importlib, torch
bt = importlib.import_module("b-tree-index-searching_b200")
n, m = %d, 1 << 27
keys = torch.arange(0, 3 * n, 3, device="cuda", dtype=torch.int32)
t = bt.Tree.build(keys, keys)
q = torch.arange(m, device="cuda", dtype=torch.int32) %% (3 * n)
out = torch.empty(m, device="cuda", dtype=torch.int32)
t.point_search(q[:1 << 22], out=out)
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
t.point_search(q, out=out)
torch.cuda.synchronize()
print("left", before - torch.cuda.mem_get_info()[0])
"""


@pytest.mark.parametrize("kb", [4, 8])
@pytest.mark.parametrize("m", [(1 << 26) + 1, 3 * (1 << 25) + 12345])
def test_every_part_is_answered(bt, cuda, kb, m):
    import torch
    it = {4: torch.int32, 8: torch.int64}[kb]
    g = torch.Generator(device=cuda)
    g.manual_seed(m)
    keys = torch.arange(0, 3 * N, 3, device=cuda, dtype=it)
    q = torch.randint(0, 3 * N + 9, (m,), generator=g, device=cuda, dtype=it)
    hit = (q % 3 == 0) & (q < 3 * N)
    want = torch.where(hit, q // 3, -1).to(it)
    with bt.Tree.build(keys, torch.arange(N, device=cuda, dtype=it)) as t:
        t.learned_train(max_error=64, iterations=10)
        for mode in ("basic", "learned"):
            v, f = t.point_search_found(q, mode=mode)
            assert torch.equal(v.view(it), want), mode
            assert torch.equal(f.bool(), hit), mode
        c = t.range_count(q, q + 30).view(torch.int64)
    below = lambda x: torch.clamp((x.to(torch.int64) + 2) // 3, max=N)  # noqa: E731
    assert torch.equal(c, below(q + 31) - below(q))


def test_scratch_of_a_large_batch_is_bounded(bt, cuda):
    """2^27 queries of 4 bytes keep no more than 2^26 queries' scratch (12 bytes
    each) and its rounding in the pool."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(bt.__file__)))
    r = subprocess.run([sys.executable, "-c", POOL % N], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    assert int(r.stdout.split("left")[1]) <= 12 * (1 << 26) + (64 << 20)
