"""How a partition pass cuts its batch (csrc/bt_part_cut.h), on devices of any
number of SMs: the positions its tables give every tile's digits, worked out
here as the kernels do, are those of a stable partition."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "b-tree-index-searching_b200", "csrc")
SHIM = """
#include "bt_part_cut.h"
extern "C" void cut(uint64_t n, uint32_t cap, uint64_t sms, uint64_t *out) {
    const bt::PartCut c = bt::part_cut(n, cap, sms);
    out[0] = c.tile; out[1] = c.per; out[2] = c.ntiles; out[3] = c.nchunks; out[4] = c.direct;
}
"""
CAPS = (8192, 6144, 4096)  # tile sizes of the item widths


@pytest.fixture(scope="module")
def cut(tmp_path_factory):
    d = tmp_path_factory.mktemp("cut")
    (d / "cut.cpp").write_text(SHIM)
    so = str(d / "cut.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", CSRC, "-o", so,
                    str(d / "cut.cpp")], check=True)
    fn = ctypes.CDLL(so).cut
    fn.argtypes = [ctypes.c_uint64, ctypes.c_uint32, ctypes.c_uint64, ctypes.c_void_p]

    def run(n, cap, sms):
        out = np.zeros(5, dtype=np.uint64)
        fn(n, cap, sms, out.ctypes.data_as(ctypes.c_void_p))
        return (int(x) for x in out)
    return run


def tile_starts(counts, per, nchunks, direct):
    """Where each tile's items of each digit go, from the tables the count
    pass writes (counts: a row per tile)."""
    ntiles = len(counts)
    chunks = np.add.reduceat(counts, np.arange(0, ntiles, per), axis=0)
    assert len(chunks) == nchunks
    tot = chunks.sum(axis=0)
    first = np.cumsum(tot) - tot
    pos = np.empty_like(counts)
    for t in range(ntiles):
        if direct:  # the rows before this CTA's, whose block index is the tile's
            pos[t] = first + chunks[:t].sum(axis=0)
        else:       # the prefix of the tile's chunk
            pos[t] = first + chunks[:t // per].sum(axis=0)
        if per > 1:
            pos[t] += counts[t - t % per:t].sum(axis=0)
    return pos


@pytest.mark.parametrize("sms", [1, 2, 7, 18, 31, 32, 36, 63, 64, 74, 148, 300])
@pytest.mark.parametrize("cap", CAPS)
def test_tiles_start_where_a_stable_partition_puts_them(cut, sms, cap):
    g = np.random.default_rng(sms)
    ctas = min(512, 2 * sms)
    sizes = {1, 1023, 1025, cap, cap + 1, 64 * cap, 64 * cap + 1, 127 * cap, ctas * 1024 + 1,
             ctas * cap, ctas * cap + 1, 2 * ctas * cap - 5, 65 * 1024, 303104, 598016}
    for n in sorted(s for s in sizes if s <= 1 << 22):
        tile, per, ntiles, nchunks, direct = cut(n, cap, sms)
        assert 0 < tile <= cap and tile % 32 == 0 and (ntiles - 1) * tile < n <= ntiles * tile
        assert nchunks <= 512 and nchunks <= ctas
        # the table of the tiles (allocated for tiles of the largest size)
        assert per == 1 or ntiles <= -(-n // cap)
        counts = g.integers(0, 5, size=(ntiles, 4))
        tot = counts.sum(axis=0)
        want = np.cumsum(tot) - tot + np.cumsum(counts, axis=0) - counts
        assert np.array_equal(tile_starts(counts, per, nchunks, direct), want), (n, per, nchunks)
