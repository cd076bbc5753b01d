"""The device sort's scratch: one copy of the pairs and its table, so that a
sort that fits beside its inputs and outputs still does."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import importlib, torch
bt = importlib.import_module("b-tree-index-searching_b200")
kb, vb, n = %d, %d, 1 << 25
it = {4: torch.int32, 8: torch.int64}
k = torch.randint(0, 1 << 31, (n,), device="cuda").to(it[kb])
v = torch.arange(n, device="cuda", dtype=it[vb])
bt.sort_pairs(k[:1000], v[:1000])
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
ok, ov = bt.sort_pairs(k, v)
torch.cuda.synchronize()
left = before - torch.cuda.mem_get_info()[0] - n * (kb + vb)
s, at = torch.sort(k, stable=True)
assert torch.equal(ok.view(it[kb]), s) and torch.equal(ov.view(it[vb]), v[at])
print("left", left)
"""


@pytest.mark.parametrize("kb,vb", [(4, 4), (4, 8), (8, 4), (8, 8)])
def test_scratch_is_one_copy(bt, cuda, kb, vb):
    n = 1 << 25
    root = os.path.dirname(os.path.dirname(os.path.abspath(bt.__file__)))
    r = subprocess.run([sys.executable, "-c", CODE % (kb, vb)], cwd=root, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    # the pairs, a table of up to a quarter of a byte a pair, allocation granularity
    assert int(r.stdout.split("left")[1]) <= n * (kb + vb) + n // 4 + (96 << 20)
