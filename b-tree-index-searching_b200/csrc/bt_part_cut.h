// How a partition pass cuts its batch (host arithmetic only; see bt_group.cu).
#pragma once

#include <stdint.h>

#include <algorithm>

namespace bt {

constexpr int kPartCtas = 2;         // CTAs per SM
constexpr int kPartMaxChunks = 512;
constexpr uint64_t kPartMinTile = 1024;  // items a CTA takes at least
constexpr uint32_t kPartDirect = 64;     // tables of up to so many rows are summed by the scatter

// Tiles of `tile` items, `per` consecutive tiles to a chunk.  direct: every
// chunk is one tile and the table of their counts is short enough for the
// scatter to sum its rows itself, the row of a CTA's one tile being its block
// index.  (A short table alone does not say so: with fewer than 64 SMs, a MIG
// slice's or an MPS limit's, 64 chunks may hold several tiles each.)
struct PartCut {
    uint64_t n;
    uint32_t tile, per, ntiles, nchunks;
    bool direct;
};

// n items (at least one) in tiles of up to `tile_cap`, a multiple of 32, on a
// device of `sms` SMs: kPartCtas CTAs per SM, one chunk each; a batch that does
// not fill them with whole tiles gets smaller ones, in whole rows of a warp.
inline PartCut part_cut(uint64_t n, uint32_t tile_cap, uint64_t sms) {
    const uint64_t ctas = std::min<uint64_t>(kPartMaxChunks, kPartCtas * std::max<uint64_t>(1, sms));
    PartCut cut;
    cut.n = n;
    cut.tile = (uint32_t)std::min<uint64_t>(
        tile_cap, std::max<uint64_t>(kPartMinTile, ((n + ctas - 1) / ctas + 31) / 32 * 32));
    cut.ntiles = (uint32_t)((n + cut.tile - 1) / cut.tile);
    cut.per = (uint32_t)((cut.ntiles + ctas - 1) / ctas);
    cut.nchunks = (cut.ntiles + cut.per - 1) / cut.per;
    cut.direct = cut.per == 1 && cut.nchunks <= kPartDirect;
    return cut;
}

}  // namespace bt
