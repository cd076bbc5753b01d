"""Rectangle counts by the code directory over points that leave stretches of
it without a key: of lengths about those of the pieces they are filled in, at
its start, between points and at its end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = (1 << 21) + 5  # a directory of 2^19 entries, 2^13 codes each


def _demorton(z):
    out = []
    for s in (0, 1):
        v = (z >> s) & 0x55555555
        for k, m in ((1, 0x33333333), (2, 0x0F0F0F0F), (4, 0x00FF00FF), (8, 0x0000FFFF)):
            v = (v | (v >> k)) & m
        out.append(v)
    return out


@pytest.mark.parametrize("gaps", [[4095, 4096, 4097, 4098], [8191, 8192, 8193, 8194], [1, 20000, 4096],
                                  [524287], [0],
                                  [30, 3000, 500000, 12289]])
@pytest.mark.parametrize("low", [0, 8191])
def test_stretches_without_points(bt, orc, cuda, gaps, low):
    import torch
    g = np.random.default_rng(sum(gaps) + low)
    at = np.cumsum(gaps)
    at = at[at < 1 << 19]
    z = np.sort((at[g.integers(0, len(at), size=N)].astype(np.int64) << 13) + low).astype(np.uint32)
    ids = g.permutation(N).astype(np.uint32)
    ids = ids[np.lexsort((ids, z))]
    nr = N // 128 + 3
    x, y = _demorton(z[g.integers(0, N, size=nr)].astype(np.int64))
    x, y = x + g.integers(-2, 3, size=nr), y + g.integers(-2, 3, size=nr)
    x0, y0 = np.clip(x - 3, 0, 65535), np.clip(y - 3, 0, 65535)
    x1, y1 = np.clip(x, 0, 65535), np.clip(y, 0, 65535)
    keep = g.random(nr) < 0.003  # boxes with many points, and empty ones
    x0, x1 = np.where(keep, x0, 7), np.where(keep, x1, 6)
    x0[0], y0[0], x1[0], y1[0] = 0, 0, 65535, 65535
    box = [a.astype(np.uint16) for a in (x0, y0, x1, y1)]
    ec, eo, ei = orc.rect_search(z, ids, *box)
    with bt.Tree.build(torch.from_numpy(z).to(cuda), torch.from_numpy(ids).to(cuda)) as t:
        c, off, got = bt.rect_search(t, *(torch.from_numpy(a).to(cuda) for a in box))
    assert np.array_equal(c.cpu().numpy(), ec)
    assert np.array_equal(off.cpu().numpy(), eo)
    assert np.array_equal(got.cpu().numpy().astype(np.uint64), ei.astype(np.uint64))
