"""Rectangle counts by the code directory: batches with few points per box,
points that crowd into a few codes, lie on the grid's corners or repeat, cells
smaller than a directory entry, and empty boxes among the others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(kind, n, g):
    if kind == "uniform":
        return g.integers(0, 1 << 16, size=n), g.integers(0, 1 << 16, size=n)
    if kind == "crowded":  # long empty stretches of the directory
        return 40000 + g.integers(0, 64, size=n), g.integers(0, 64, size=n)
    x, y = g.choice([0, 1, 32767, 32768, 65534, 65535], size=(2, n))  # repeated points at corners
    return x, y


@pytest.mark.parametrize("kind", ["uniform", "crowded", "corners"])
@pytest.mark.parametrize("n,vt", [(1, np.uint32), (1000, np.uint64), (70001, np.uint32), (300007, np.uint32)])
@pytest.mark.parametrize("side", [1, 20, 300, 65536])
def test_directory_counts_match_the_oracle(bt, orc, wl, cuda, kind, n, vt, side):
    import torch
    g = np.random.default_rng(n + side)
    x, y = (a.astype(np.uint16) for a in _points(kind, n, g))
    z = wl.morton_u16(x, y)
    ids = g.permutation(n).astype(vt)
    o = np.lexsort((ids, z))
    zs, idss = z[o], ids[o]
    nr = 2999 if side < 1000 or n < 2000 else 300 if n < 80000 else 0
    nr = max(nr, n // 128 + 1)  # the directory's rule
    if side > 1000 and n > 80000:
        pytest.skip("every box holds every point")
    ax = x[g.integers(0, n, size=nr)].astype(np.int64) - g.integers(0, side, size=nr)
    ay = y[g.integers(0, n, size=nr)].astype(np.int64) - g.integers(0, side, size=nr)
    x0, y0 = np.clip(ax, 0, 65535), np.clip(ay, 0, 65535)
    x1 = np.minimum(x0 + g.integers(0, side, size=nr), 65535)
    y1 = np.minimum(y0 + g.integers(0, side, size=nr), 65535)
    x0[::17], x1[::17] = 9, 8  # empty boxes
    box = [a.astype(np.uint16) for a in (x0, y0, x1, y1)]
    ec, eo, ei = orc.rect_search(zs, idss.astype(np.uint32), *box)
    with bt.Tree.build(torch.from_numpy(zs).to(cuda), torch.from_numpy(idss).to(cuda)) as t:
        for mode in ("basic", "zorder"):
            c, off, got = bt.rect_search(t, *(torch.from_numpy(a).to(cuda) for a in box), mode=mode)
            assert np.array_equal(c.cpu().numpy(), ec), mode
            assert np.array_equal(off.cpu().numpy(), eo), mode
            assert np.array_equal(got.cpu().numpy().astype(np.uint64), ei.astype(np.uint64)), mode
