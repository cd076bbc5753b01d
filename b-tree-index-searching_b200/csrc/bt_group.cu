// Query grouping, device sort, bucket order, exclusive scan and range-ID fill.
//
// Grouping reorders a query batch so that queries that walk the same part of
// the tree run next to each other (in the same CTAs, at the same time), which
// turns repeated node and leaf-sector reads into L1/L2 hits.  The reference
// does this with an MSD radix partition by 8-bit digits, iterated until every
// group holds at most GROUP_SEARCH_SIZE = 33,000 queries, with a host round
// trip per pass and per group (genGrouping, grouping.cu:1677-1851;
// radixGroupGPU :776; radixGroupSingleKernelGPU :1288), and one CTA per group.
//
// Here a group key of D bits is computed per query and the batch is sorted by
// it with D/8 stable LSD counting passes (count -> prefix -> scatter), all
// on the device with no host round trip.  Each scatter carries the caller's
// index, so results are written straight back in the caller's order.  (Large
// batches take the unstable one-pass bucket order below instead.)
//   point : the top D bits of the key (relative to the tree's key width);
//   2D    : (top D/2 bits of start, top D/2 bits of end), row-major -- a true
//           2-D cell, where the reference buckets by the product of two
//           digits (bucketIdentify2d, grouping2d.cu:24-31);
//   Z     : the Morton interleave of those two D/2-bit coordinates, as the
//           reference interleaves start and end (calcuateZorder2d,
//           zOrder2d.cu:27-54) before grouping by the code.
// A pass is stable, so the order is deterministic (the reference's in-block
// atomicAdd scatter is not, grouping.cu:451-452).
#include <algorithm>
#include <atomic>
#include <type_traits>
#include <vector>

#include "bt_part_cut.h"
#include "bt_search.cuh"
#include "bt_sort.cuh"

namespace bt {
namespace {

struct GroupKeyParams {
    int kind;   // PartitionKind
    int shift;  // right shift applied to keys
    int cbits;  // bits per coordinate (2D/Z) or total bits (point)
};

__device__ __forceinline__ uint32_t spread16(uint32_t x) {
    x &= 0xFFFFu;
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}

template <typename K>
__device__ __forceinline__ uint32_t group_key(K a, K b, const GroupKeyParams &p) {
    if (p.kind == kPartRadix) return (uint32_t)((uint64_t)a >> p.shift);  // caller takes the low byte
    const uint64_t lim = (1ull << p.cbits) - 1;
    uint64_t x = (uint64_t)a >> p.shift;
    x = x < lim ? x : lim;
    if (p.kind == kPartPoint) return (uint32_t)x;
    uint64_t y = (uint64_t)b >> p.shift;
    y = y < lim ? y : lim;
    if (p.kind == kPart2D) return (uint32_t)((x << p.cbits) | y);
    return spread16((uint32_t)x) | (spread16((uint32_t)y) << 1);
}

// ------------------------------------------------------------ partition ----
//
// One stable partition by an 8-bit digit.  The batch is cut into tiles, and
// runs of consecutive tiles into one chunk per resident CTA:
//   part_count_kernel    counts the digits chunk by chunk (and how many of
//                        the chunk's come before each of its tiles);
//   part_prefix_kernel   turns the chunk counts into exclusive prefixes over
//                        the chunks, and the digit totals (small tables are
//                        summed by the next kernel itself);
//   part_scatter_kernel  ranks a tile's items, orders them in shared memory
//                        and writes them out digit by digit.  The tiles in
//                        flight are consecutive ones, so what they write for
//                        a digit is one stretch.
// The keys are read twice, but no tile waits for another: a single pass with
// decoupled look-back (Merrill & Garland 2016) walked back over most of the
// hundreds of tiles in flight.  u32 pairs, 2^26: 1.09 ms a pass with the
// look-back, 0.46 ms here (count 0.075, scatter 0.38; 1.3 GB, 0.2 ms at the
// copy rate).  What bounds the scatter: 102 warp instructions a row of 32
// items, most of them on the half-rate integer pipe, and 22 shared-memory
// wavefronts (32 warps per SM between barriers).  Smaller tiles
// with three CTAs per SM: 0.47 ms; 256-thread CTAs: 0.51 and more.
constexpr int kPT = 512;             // partition threads per CTA
constexpr int kPWarps = kPT / 32;

// Items per thread of a tile, as many as two CTAs per SM have registers (64 a
// thread) and shared memory for: a tile's stretch of a digit gets longer.
// Whole sorts at 2^26, items per thread 8 / 12 / 16: u32 pairs 1.93 / 1.80 /
// 1.78 ms, u64 pairs 5.8 / 7.2 / 7.3 ms (with votes 0.07 ms faster than now's).
template <int ITEM_BYTES>
__host__ __device__ constexpr int part_ipt() {
    return ITEM_BYTES <= 8 ? 16 : ITEM_BYTES <= 12 ? 12 : 8;
}

// Source and destination of one pass.  b only for two-key items; p_in may be
// null (the item's index is its payload).
template <typename K, typename P>
struct PassIO {
    const K *a_in, *b_in;
    const P *p_in;
    K *a_out, *b_out;
    P *p_out;
};

// The sort's buffers: the passes go back and forth between the output and one
// copy, so that the last one ends in the output.  `vary` has a bit set where some
// key differs from the first one: a pass whose digit has no such bit would change
// nothing and is skipped (pass 0, which fills vary in, never is), so which of the
// two a pass writes depends on how many run after it.
template <typename K, typename P>
struct SortIO {
    const K *in;
    const P *p_in;
    K *tk, *out;
    P *tp, *p_out;
    unsigned long long *vary;
    int passes;
};

// True when pass p runs; io receives its buffers (the count of pass 0, which
// is still filling vary in, only uses the source).
template <typename K, typename P>
__device__ __forceinline__ bool sort_pass(const SortIO<K, P> &s, int p, PassIO<K, P> &io) {
    const unsigned long long v = *s.vary | 0xFFull;
    if (((v >> (8 * p)) & 0xFFull) == 0) return false;
    int before = 0, after = 0;
    for (int k = 0; k < s.passes; k++) {
        const bool runs = ((v >> (8 * k)) & 0xFFull) != 0;
        before += k < p && runs;
        after += k > p && runs;
    }
    const bool to_out = (after & 1) == 0;  // the pass before it, if any, wrote the other one
    io.a_in = before == 0 ? s.in : to_out ? s.tk : s.out;
    io.p_in = before == 0 ? s.p_in : to_out ? s.tp : s.p_out;
    io.a_out = to_out ? s.out : s.tk;
    io.p_out = to_out ? s.p_out : s.tp;
    io.b_in = nullptr;
    io.b_out = nullptr;
    return true;
}

// Digit of pass p of an item: byte p of its group key (of the key itself for
// the radix sort).  KEY: a sort's, known at compile time (2^25 u64 pairs 2.13 ->
// 2.08 ms; where a tile has more than eight items a thread nvcc then takes the
// votes of later rows ahead and spills: u32 pairs, 2^26, 1.85 -> 2.15).
template <typename K, bool KEY>
__device__ __forceinline__ uint32_t pass_digit(K a, K b, const GroupKeyParams &gp, int p) {
    if (KEY || gp.kind == kPartRadix) return (uint32_t)(a >> (8 * p)) & 0xFFu;
    return (group_key<K>(a, b, gp) >> (8 * p)) & 0xFFu;
}

// Row c of chunk_tab: the digits of chunk c.  Row t of tile_tab (when a chunk
// has several tiles): those of the chunk's tiles before tile t.  Counters per
// warp in shared memory (atomics only collide inside a warp).
template <typename K, typename P, bool HAS_B, bool SORT, typename IO>
__global__ void __launch_bounds__(kPT)
part_count_kernel(const __grid_constant__ IO io_in, const __grid_constant__ PartCut cut,
                  GroupKeyParams gp, int pass, uint32_t *__restrict__ chunk_tab,
                  uint32_t *__restrict__ tile_tab) {
    __shared__ uint32_t h[kPWarps][256];
    __shared__ unsigned long long s_vary;
    PassIO<K, P> io;
    if constexpr (SORT) {
        if (!sort_pass<K, P>(io_in, pass, io)) return;
    } else {
        io = io_in;
    }
    const K *__restrict__ a = io.a_in;
    const K *__restrict__ b = io.b_in;
    for (int i = threadIdx.x; i < kPWarps * 256; i += kPT) (&h[0][0])[i] = 0;
    if (threadIdx.x == 0) s_vary = 0;
    uint32_t *hw = h[threadIdx.x >> 5];
    K diff = 0;
    const K first = SORT && pass == 0 ? a[0] : (K)0;
    uint32_t run = 0;  // digit threadIdx.x in the chunk so far
    const uint32_t t0 = blockIdx.x * cut.per, t1 = min(cut.ntiles, t0 + cut.per);
    for (uint32_t t = t0; t < t1; t++) {
        __syncthreads();
        const uint64_t c0 = (uint64_t)t * cut.tile, c1 = min(cut.n, c0 + cut.tile);
        constexpr int U = 8;  // loads in flight per thread
        uint64_t i = c0 + threadIdx.x;
        for (; i + (U - 1) * kPT < c1; i += U * kPT) {
            K av[U], bv[U];
#pragma unroll
            for (int j = 0; j < U; j++) {
                av[j] = a[i + j * kPT];
                bv[j] = HAS_B ? b[i + j * kPT] : (K)0;
            }
#pragma unroll
            for (int j = 0; j < U; j++) {
                atomicAdd(&hw[pass_digit<K, SORT>(av[j], bv[j], gp, pass)], 1u);
                if (SORT) diff |= av[j] ^ first;
            }
        }
        for (; i < c1; i += kPT) {
            const K av = a[i];
            atomicAdd(&hw[pass_digit<K, SORT>(av, HAS_B ? b[i] : (K)0, gp, pass)], 1u);
            if (SORT) diff |= av ^ first;
        }
        if (tile_tab && threadIdx.x < 256) tile_tab[t * 256u + threadIdx.x] = run;
        __syncthreads();
        if (threadIdx.x < 256) {
#pragma unroll
            for (int w = 0; w < kPWarps; w++) {
                run += h[w][threadIdx.x];
                h[w][threadIdx.x] = 0;
            }
        }
    }
    if (threadIdx.x < 256) chunk_tab[blockIdx.x * 256u + threadIdx.x] = run;
    if constexpr (SORT) {
        if (pass == 0) {
            if (diff) atomicOr(&s_vary, (unsigned long long)diff);
            __syncthreads();
            if (threadIdx.x == 0 && s_vary) atomicOr(io_in.vary, s_vary);
        }
    }
}

// Column d of the table (one warp per digit) -> exclusive prefix over the
// rows; its sum goes to row `rows`.  A lane takes consecutive rows, all its
// loads in flight.
__global__ void __launch_bounds__(256)
part_prefix_kernel(uint32_t *__restrict__ table, int rows) {
    constexpr int R = kPartMaxChunks / 32;
    const int d = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int per = (rows + 31) / 32;
    uint32_t v[R], sum = 0;
#pragma unroll
    for (int k = 0; k < R; k++) {
        const int r = lane * per + k;
        v[k] = k < per && r < rows ? table[r * 256 + d] : 0u;
        sum += v[k];
    }
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    uint32_t run = x - sum;
#pragma unroll
    for (int k = 0; k < R; k++) {
        const int r = lane * per + k;
        if (k < per && r < rows) table[r * 256 + d] = run;
        run += v[k];
    }
    if (lane == 31) table[rows * 256 + d] = x;
}

// Exclusive scan of the values of threads 0-255; warp_tot is 8 words.  Every
// thread of the CTA calls it (one barrier; another one has to pass before
// the next call).
__device__ __forceinline__ uint32_t block_exscan256(uint32_t v, uint32_t *warp_tot) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
    if (w < 8) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[w] = x;
    }
    __syncthreads();
    uint32_t wp = 0;
    if (w < 8) {
#pragma unroll
        for (int k = 0; k < 8; k++) wp += k < w ? warp_tot[k] : 0u;
    }
    return x - v + wp;
}

template <typename K, typename P, bool HAS_B>
struct PartSmem {
    static constexpr int IPT = part_ipt<(int)(sizeof(K) * (HAS_B ? 2 : 1) + sizeof(P))>();
    static constexpr int T = kPT * IPT;  // items per tile
    // key and payload of one width go through shared memory as one record
    static constexpr bool REC = !HAS_B && sizeof(K) == sizeof(P);
    struct alignas(sizeof(K) * 2) Rec {
        K a;
        P p;
    };
    static constexpr size_t bytes = kPWarps * 256 * sizeof(uint32_t) + 256 * sizeof(uint32_t) +
                                    (size_t)T * (sizeof(K) * (HAS_B ? 2 : 1) + sizeof(P));
};

// The lanes whose 8-bit digit equals this lane's, among those with `valid`
// (0 for the others): a vote per bit, from which every lane whose bit is another
// is dropped (vote xor this lane's bit in all places).  The whole sort of 2^26 u32
// pairs: 3.05 ms with __match_any_sync, whose time grows with the number of
// distinct digits, 1.95 with a shared-memory word per digit that lanes set their
// bit in (conflicts), 1.93 with the bit made a mask by a subtraction, 2.03 with a
// branch on it, 1.85 like this.
template <bool ALL>
__device__ __forceinline__ unsigned same_digit(uint32_t d, bool valid) {
    unsigned m = ALL ? 0xffffffffu : __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const int mine = (int)(d << (31 - b)) >> 31;  // this lane's bit in all 32 places
        m &= ~(__ballot_sync(0xffffffffu, mine < 0) ^ (unsigned)mine);
    }
    return m;
}

template <typename K, typename P, bool HAS_B, bool SORT, typename IO>
__global__ void __launch_bounds__(kPT, kPartCtas)
part_scatter_kernel(const __grid_constant__ IO io_in, const __grid_constant__ PartCut cut,
                    GroupKeyParams gp, int pass, const uint32_t *__restrict__ chunk_tab,
                    const uint32_t *__restrict__ tile_tab) {
    using PS = PartSmem<K, P, HAS_B>;
    constexpr int IPT = PS::IPT;
    constexpr uint32_t T = PS::T;
    constexpr bool KEY = SORT && IPT <= 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t warp_tot[8];
    uint32_t(*cnt)[256] = reinterpret_cast<uint32_t(*)[256]>(smem_raw);
    uint32_t *gbase = reinterpret_cast<uint32_t *>(cnt + kPWarps);
    // the ordered tile: a record per item, or an array per field
    using Rec = typename PS::Rec;
    Rec *sr = reinterpret_cast<Rec *>(gbase + 256);
    K *sa = reinterpret_cast<K *>(gbase + 256);
    K *sb = sa + (HAS_B ? T : 0);
    P *sp = reinterpret_cast<P *>(sb + T);
    PassIO<K, P> io;
    if constexpr (SORT) {
        if (!sort_pass<K, P>(io_in, pass, io)) return;
    } else {
        io = io_in;
    }
    const K *__restrict__ a = io.a_in;
    const K *__restrict__ b = io.b_in;
    const P *__restrict__ pin = io.p_in;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t rows = cut.nchunks;

    // where the batch's items of digit `threadIdx.x` start (for a direct cut
    // also where this CTA's one tile puts its own)
    uint32_t first = 0;
    {
        uint32_t tot = 0, pre = 0;
        if (threadIdx.x < 256) {
            if (!cut.direct) {
                tot = chunk_tab[rows * 256u + threadIdx.x];
            } else {
#pragma unroll 8
                for (uint32_t r = 0; r < rows; r++) {
                    const uint32_t v = chunk_tab[r * 256u + threadIdx.x];
                    pre += r < blockIdx.x ? v : 0u;
                    tot += v;
                }
            }
        }
        first = block_exscan256(tot, warp_tot) + pre;
    }
    uint32_t *cw = cnt[w];
    K av[IPT], bv[HAS_B ? IPT : 1];
    uint32_t rpw = 0;  // rows of 32 items per warp: IPT, or fewer in a short tile
    auto tile_items = [&](uint32_t t) {
        return (uint32_t)min((uint64_t)cut.tile, cut.n - (uint64_t)t * cut.tile);
    };
    auto load_keys = [&](uint32_t t) {
        const uint64_t t0 = (uint64_t)t * cut.tile;
        const uint32_t tn = tile_items(t);
        rpw = tn == T ? (uint32_t)IPT : (tn + kPT - 1) / kPT;
#pragma unroll
        for (int j = 0; j < IPT; j++) {
            const uint32_t i = (w * rpw + j) * 32 + lane;
            const bool v = tn == T || (j < (int)rpw && i < tn);
            av[j] = v ? a[t0 + i] : (K)0;
            if (HAS_B) bv[j] = v ? b[t0 + i] : (K)0;
        }
    };
    const unsigned lt = (1u << lane) - 1u;
    // One tile: FULL has every item (no bounds to check).
    auto tile = [&](auto full_tag, uint32_t t, uint32_t tn) {
        constexpr bool FULL = decltype(full_tag)::value;
        const uint64_t t0 = (uint64_t)t * cut.tile;
        const uint32_t r0 = w * (FULL ? (uint32_t)IPT : rpw) * 32 + lane;  // the lane's first item
        auto live = [&](int j) { return FULL || (j < (int)rpw && r0 + j * 32 < tn); };
#pragma unroll
        for (int k = 0; k < 2; k++) reinterpret_cast<uint4 *>(cw)[k * 32 + lane] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        // Stable rank of every item among the same-digit items of its warp
        // (item order = row, then lane).
        uint32_t rk[IPT];
#pragma unroll
        for (int j = 0; j < IPT; j++) {
            const bool v = live(j);
            const uint32_t d = pass_digit<K, KEY>(av[j], HAS_B ? bv[j] : (K)0, gp, pass);
            const unsigned m = same_digit<FULL>(d, v);
            const uint32_t c = v ? cw[d] : 0u;
            const uint32_t below = __popc(m & lt);
            __syncwarp();
            if (v && below == 0) cw[d] = c + __popc(m);
            __syncwarp();
            rk[j] = c + below;
        }
        // the payload arrives while the digits are scanned
        P pv[IPT];
#pragma unroll
        for (int j = 0; j < IPT; j++) {
            const uint64_t i = t0 + r0 + j * 32;
            pv[j] = pin ? (live(j) ? pin[i] : (P)0) : (P)i;
        }
        uint32_t run = first;  // where the tile's first item of digit `threadIdx.x` goes
        if (threadIdx.x < 256) {
            if (!cut.direct) run += chunk_tab[(t / cut.per) * 256u + threadIdx.x];
            if (tile_tab) run += tile_tab[t * 256u + threadIdx.x];
        }
        __syncthreads();
        // per digit: the tile's total, then every warp's first slot
        uint32_t tot = 0;
        if (threadIdx.x < 256) {
#pragma unroll
            for (int k = 0; k < kPWarps; k++) tot += cnt[k][threadIdx.x];
        }
        const uint32_t start = block_exscan256(tot, warp_tot);
        if (threadIdx.x < 256) {
            uint32_t x = start;
#pragma unroll
            for (int k = 0; k < kPWarps; k++) {
                const uint32_t c = cnt[k][threadIdx.x];
                cnt[k][threadIdx.x] = x;
                x += c;
            }
            gbase[threadIdx.x] = run - start;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IPT; j++) {
            if (live(j)) {
                const uint32_t d = pass_digit<K, KEY>(av[j], HAS_B ? bv[j] : (K)0, gp, pass);
                const uint32_t lp = cw[d] + rk[j];
                if constexpr (PS::REC) {
                    sr[lp] = Rec{av[j], pv[j]};
                } else {
                    sa[lp] = av[j];
                    if (HAS_B) sb[lp] = bv[j];
                    sp[lp] = pv[j];
                }
            }
        }
        __syncthreads();
        if (t + gridDim.x < cut.ntiles) load_keys(t + gridDim.x);  // these arrive behind the writes
        auto put = [&](uint32_t lp) {
            K ka, kb = 0;
            P kp;
            if constexpr (PS::REC) {
                const Rec r = sr[lp];
                ka = r.a;
                kp = r.p;
            } else {
                ka = sa[lp];
                if (HAS_B) kb = sb[lp];
                kp = sp[lp];
            }
            const uint32_t g = gbase[pass_digit<K, KEY>(ka, kb, gp, pass)] + lp;
            io.a_out[g] = ka;
            if (HAS_B) io.b_out[g] = kb;
            io.p_out[g] = kp;
        };
        if constexpr (FULL) {
#pragma unroll
            for (int j = 0; j < IPT; j++) put(j * kPT + threadIdx.x);
        } else {
            for (uint32_t lp = threadIdx.x; lp < tn; lp += kPT) put(lp);
        }
        // no barrier here: the next tile writes gbase and the ordered items
        // only after its first one
    };
    if (blockIdx.x < cut.ntiles) load_keys(blockIdx.x);
    for (uint32_t t = blockIdx.x; t < cut.ntiles; t += gridDim.x) {
        const uint32_t tn = tile_items(t);
        if (tn == T) tile(std::true_type{}, t, T);
        else tile(std::false_type{}, t, tn);
    }
}

// -------------------------------------------------------------- buckets ----
//
// The order a large point batch is searched in: by bucket, in any order
// inside one, so that the queries near each other in time are near each other
// in the tree.  One pass of up to 2,048 buckets:
//   bucket_count_kernel    batch counts of every bucket;
//   bucket_start_kernel    their exclusive scan (the buckets' cursors), and
//                          the leaf block where each bucket's keys start;
//   bucket_scatter_kernel  orders a tile in shared memory, reserves each
//                          bucket's part of the output at its cursor and
//                          writes the tile out bucket by bucket; pos[i] = the
//                          slot query i went to;
//   bucket_gather_kernel   (after the search) out[i] = the result in slot
//                          pos[i].
// Results are written to the slots and gathered back, not scattered by the
// search: a scattered 8-byte write costs DRAM a 32-byte write and a 64-byte
// read (2^24 u64 results: 0.53 GB written, 1 GB read), while the gather's
// tile finds its results in runs, as the scatter's tile left them.
// The order need not be stable (no caller sees it), so an item's rank is what
// a shared-memory atomic returns: 11 bits in one pass, where the stable
// partition takes a vote per bit and two passes.

constexpr int kBT = 512;
template <typename K>
struct BucketSmem {
    static constexpr int IPT = sizeof(K) == 4 ? 16 : 12;
    static constexpr int T = kBT * IPT;
    static constexpr size_t bytes = (size_t)T * sizeof(K) + 2 * kMaxBuckets * sizeof(uint32_t);
};

// Query i of a batch.  A range batch is two batches of lower bounds, lo[i]
// and then hi[i] + 1 (the bound of an hi at the largest value is not used).
template <typename K>
struct PointBatch {
    const K *q;
    __device__ __forceinline__ K get(uint64_t i) const { return q[i]; }
};
template <typename K>
struct RangeBatch {
    const K *lo, *hi;
    uint64_t nr;
    __device__ __forceinline__ K get(uint64_t i) const { return i < nr ? lo[i] : (K)(hi[i - nr] + 1); }
};

template <typename K, typename B>
__global__ void __launch_bounds__(kBT)
bucket_count_kernel(const __grid_constant__ B q, uint64_t n, const __grid_constant__ BucketMap map,
                    uint32_t *__restrict__ total) {
    constexpr int C = kMaxBuckets <= 2048 ? 4 : kMaxBuckets <= 4096 ? 2 : 1;  // copies
    __shared__ uint32_t h[C][kMaxBuckets];
    const int nb = (int)map.last + 1;
    for (int i = threadIdx.x; i < C * kMaxBuckets; i += kBT) (&h[0][0])[i] = 0;
    __syncthreads();
    uint32_t *hw = h[(threadIdx.x >> 5) & (C - 1)];
    constexpr int U = 8;
    const uint64_t step = (uint64_t)gridDim.x * kBT * U;
    for (uint64_t i0 = (uint64_t)blockIdx.x * kBT * U + threadIdx.x; i0 < n; i0 += step) {
        K v[U];
#pragma unroll
        for (int j = 0; j < U; j++) v[j] = i0 + j * kBT < n ? q.get(i0 + j * kBT) : (K)0;
#pragma unroll
        for (int j = 0; j < U; j++)
            if (i0 + j * kBT < n) atomicAdd(&hw[map.of(v[j])], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += kBT) {
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < C; k++) c += h[k][i];
        if (c) atomicAdd(&total[i], c);
    }
}

// Block 0: start = cursor = exclusive scan of total (start[nb] = n), and the
// search's work items: every bucket's queries in equal slices of at most `slice`
// (item = bucket, first query, queries).  The others: first[b] =
// leaf block of the first key at or above bucket b's first key (b = nb: of the
// first key equal to the largest), so the first key at or above a query of
// bucket b lies in blocks first[b] .. first[b + 1], at most bucket_blocks ones.
template <typename K>
__global__ void __launch_bounds__(1024)
bucket_start_kernel(const __grid_constant__ DevTree t, const __grid_constant__ BucketMap map, uint32_t slice,
                    const uint32_t *__restrict__ total, uint32_t *__restrict__ cursor,
                    uint32_t *__restrict__ first, uint4 *__restrict__ items,
                    uint32_t *__restrict__ n_items) {
    const uint32_t nb = map.last + 1;
    if (blockIdx.x > 0) {  // eight lanes per bucket
        const uint32_t i = ((blockIdx.x - 1) * blockDim.x + threadIdx.x) >> 3;
        const uint64_t k = i < nb ? map.first_key(i) : t.max_key;
        const K qe[1] = {k < t.max_key ? (K)k : (K)t.max_key};
        const bool up[1] = {false};
        uint32_t node[1] = {0};
        const int lane = threadIdx.x & 31;
        walk_from<K, 8, 1>(t, 0, qe, up, node, lane >> 3, lane & 7);
        if ((lane & 7) == 0 && i <= nb) first[i] = node[0];
        return;
    }
    constexpr int PER = kMaxBuckets / 1024;  // buckets per thread
    __shared__ uint32_t s_w[2][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t i = PER * threadIdx.x;
    uint32_t c[PER], sl[PER], cs = 0, ss = 0;
#pragma unroll
    for (int k = 0; k < PER; k++) {
        c[k] = i + k < nb ? total[i + k] : 0u;
        sl[k] = (c[k] + slice - 1) / slice;
        cs += c[k];
        ss += sl[k];
    }
    uint32_t x = cs, y = ss;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, x, o), b = __shfl_up_sync(0xffffffffu, y, o);
        if (lane >= o) {
            x += a;
            y += b;
        }
    }
    if (lane == 31) {
        s_w[0][w] = x;
        s_w[1][w] = y;
    }
    __syncthreads();
    x -= cs;
    y -= ss;
    for (int k = 0; k < w; k++) {
        x += s_w[0][k];
        y += s_w[1][k];
    }
#pragma unroll
    for (int k = 0; k < PER; k++) {
        if (i + k < nb) cursor[i + k] = x;
        const uint32_t len = sl[k] ? (c[k] + sl[k] - 1) / sl[k] : 0u;
        for (uint32_t z = 0; z < sl[k]; z++)
            items[y + z] = make_uint4(i + k, x + z * len, min(len, c[k] - z * len), 0u);
        x += c[k];
        y += sl[k];
    }
    if (threadIdx.x == blockDim.x - 1) *n_items = y;
}

// *blocks = the most leaf blocks a bucket's keys touch (eight lanes per
// bucket).  Takes the key range from the first and last key itself, so that a
// build need not wait for them first; leaves at once when *unsorted has bit 0
// set (the walk needs ascending separators).
template <typename K>
__global__ void __launch_bounds__(256)
bucket_blocks_kernel(const __grid_constant__ DevTree t, const K *__restrict__ first_key,
                     const K *__restrict__ last_key, const unsigned int *__restrict__ unsorted,
                     uint32_t *__restrict__ blocks) {
    if (unsorted && (*unsorted & 1u)) return;
    const K tmax = *last_key;
    const BucketMap map = bucket_map((uint64_t)*first_key, (uint64_t)tmax);
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int lane = threadIdx.x & 31;
    const uint32_t b = i <= map.last ? i : map.last;
    const uint64_t a = map.first_key(b), z = b == map.last ? (uint64_t)tmax : map.first_key(b + 1);
    const K qe[2] = {a < (uint64_t)tmax ? (K)a : tmax, z < (uint64_t)tmax ? (K)z : tmax};
    const bool up[2] = {false, false};
    uint32_t node[2] = {0, 0};
    walk_from<K, 8, 2>(t, 0, qe, up, node, lane >> 3, lane & 7);
    const uint32_t m = __reduce_max_sync(0xffffffffu, node[1] - node[0] + 1u);
    if (lane == 0) atomicMax(blocks, m);
}

template <typename K, typename B>
__global__ void __launch_bounds__(kBT, 2)
bucket_scatter_kernel(const __grid_constant__ B q, uint64_t n, const __grid_constant__ BucketMap map,
                      uint32_t *__restrict__ cursor, K *__restrict__ oq, uint32_t *__restrict__ pos) {
    using BS = BucketSmem<K>;
    constexpr int IPT = BS::IPT;
    constexpr uint32_t T = BS::T;
    constexpr int PER = kMaxBuckets / kBT;  // buckets per thread
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t s_w[kBT / 32];
    K *sq = reinterpret_cast<K *>(smem_raw);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(sq + T);  // counts, then each bucket's first slot
    uint32_t *gbase = cnt + kMaxBuckets;  // output slot of the tile's slot 0, per bucket
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t ntiles = (n + T - 1) / T;
    for (uint64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const uint64_t t0 = t * T;
        const uint32_t tn = (uint32_t)min((uint64_t)T, n - t0);
        K v[IPT];
        uint32_t rk[IPT];  // rank in the bucket, and the bucket above it
#pragma unroll
        for (int j = 0; j < IPT; j++) {
            const uint32_t i = j * kBT + threadIdx.x;
            v[j] = i < tn ? q.get(t0 + i) : (K)0;
        }
        for (uint32_t i = threadIdx.x; i < kMaxBuckets; i += kBT) cnt[i] = 0;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IPT; j++) {
            const uint32_t b = map.of(v[j]);
            rk[j] = b << 16;
            if (j * kBT + threadIdx.x < tn) rk[j] |= atomicAdd(&cnt[b], 1u);
        }
        __syncthreads();
        // the tile's part of every bucket, reserved (neighbouring lanes take
        // neighbouring cursors: one request a line)
#pragma unroll
        for (int k = 0; k < PER; k++) {
            const uint32_t b = k * kBT + threadIdx.x, c = cnt[b];
            gbase[b] = c ? atomicAdd(&cursor[b], c) : 0u;
        }
        // exclusive scan over the buckets, PER consecutive ones per thread
        uint32_t c[PER], sum = 0;
#pragma unroll
        for (int k = 0; k < PER; k++) {
            c[k] = cnt[threadIdx.x * PER + k];
            sum += c[k];
        }
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_w[w] = x;
        __syncthreads();
        uint32_t run = x - sum;
#pragma unroll
        for (int k = 0; k < kBT / 32; k++) run += k < w ? s_w[k] : 0u;
#pragma unroll
        for (int k = 0; k < PER; k++) {
            cnt[threadIdx.x * PER + k] = run;
            gbase[threadIdx.x * PER + k] -= run;
            run += c[k];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IPT; j++) {
            const uint32_t i = j * kBT + threadIdx.x;
            if (i < tn) {
                const uint32_t b = rk[j] >> 16;
                const uint32_t lp = cnt[b] + (rk[j] & 0xFFFFu);
                sq[lp] = v[j];
                pos[t0 + i] = gbase[b] + lp;
            }
        }
        __syncthreads();
#pragma unroll 4
        for (uint32_t lp = threadIdx.x; lp < tn; lp += kBT) {
            const K k = sq[lp];
            oq[gbase[map.of(k)] + lp] = k;
        }
        __syncthreads();
    }
}

// out[i] = res[pos[i]] (and the found flags).
template <typename V>
__global__ void __launch_bounds__(512)
bucket_gather_kernel(const V *__restrict__ res, const uint8_t *__restrict__ rfound,
                     const uint32_t *__restrict__ pos, uint64_t n, V *__restrict__ out,
                     uint8_t *__restrict__ found) {
    constexpr int U = 8;
    const uint64_t i0 = (uint64_t)blockIdx.x * (512 * U) + threadIdx.x;
    uint32_t p[U];
#pragma unroll
    for (int j = 0; j < U; j++) p[j] = i0 + j * 512 < n ? pos[i0 + j * 512] : 0u;
    V v[U];
#pragma unroll
    for (int j = 0; j < U; j++) v[j] = res[p[j]];
#pragma unroll
    for (int j = 0; j < U; j++)
        if (i0 + j * 512 < n) out[i0 + j * 512] = v[j];
    if (found) {
        uint8_t f[U];
#pragma unroll
        for (int j = 0; j < U; j++) f[j] = rfound[p[j]];
#pragma unroll
        for (int j = 0; j < U; j++)
            if (i0 + j * 512 < n) found[i0 + j * 512] = f[j];
    }
}

// counts[i] = keys in [lo[i], hi[i]] from the two bounds' ranks, and the
// lower bounds when lb is not null.
template <typename K>
__global__ void __launch_bounds__(512)
range_gather_kernel(const uint32_t *__restrict__ rank, const uint32_t *__restrict__ pos,
                    const K *__restrict__ lo, const K *__restrict__ hi, uint64_t nr, K tmax, uint64_t n,
                    uint64_t *__restrict__ counts, uint64_t *__restrict__ lb) {
    constexpr int U = 4;
    const uint64_t i0 = (uint64_t)blockIdx.x * (512 * U) + threadIdx.x;
    K a[U], b[U];
    uint32_t pa[U], pb[U];
#pragma unroll
    for (int j = 0; j < U; j++) {
        const uint64_t i = i0 + j * 512 < nr ? i0 + j * 512 : 0;
        a[j] = lo[i];
        b[j] = hi[i];
        pa[j] = pos[i];
        pb[j] = pos[nr + i];
    }
    uint64_t ra[U], rb[U];
#pragma unroll
    for (int j = 0; j < U; j++) {
        ra[j] = rank[pa[j]];
        rb[j] = rank[pb[j]];
    }
#pragma unroll
    for (int j = 0; j < U; j++) {
        if (a[j] > tmax) ra[j] = n;
        if (b[j] >= tmax) rb[j] = n;
        if (i0 + j * 512 < nr) {
            counts[i0 + j * 512] = a[j] <= b[j] && rb[j] > ra[j] ? rb[j] - ra[j] : 0;
            if (lb) lb[i0 + j * 512] = ra[j];
        }
    }
}

// ---------------------------------------------------------------- scan ----

constexpr int kST = 512;
constexpr int kSIPT = 8;
constexpr int kSTile = kST * kSIPT;

template <typename T>
__device__ __forceinline__ T block_exscan(T v, T *s_warp, T *total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[w] = x;
    __syncthreads();
    if (w == 0) {
        T y = lane < (kST / 32) ? s_warp[lane] : (T)0;
        T z = y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            T u = __shfl_up_sync(0xffffffffu, z, o);
            if (lane >= o) z += u;
        }
        if (lane < (kST / 32)) s_warp[lane] = z - y;
        if (lane == 31) *total = z;
    }
    __syncthreads();
    return x - v + s_warp[w];
}

template <typename T>
__global__ void __launch_bounds__(kST) scan_reduce_kernel(const T *__restrict__ in, uint64_t n,
                                                          T *__restrict__ sums) {
    __shared__ T s_warp[kST / 32];
    __shared__ T total;
    const uint64_t t0 = (uint64_t)blockIdx.x * kSTile + (uint64_t)threadIdx.x * kSIPT;
    T acc = 0;
#pragma unroll
    for (int j = 0; j < kSIPT; j++)
        if (t0 + j < n) acc += in[t0 + j];
    block_exscan<T>(acc, s_warp, &total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// total_max (optional): [0] = sum of the inputs, [1] (zeroed before) = the
// largest.
template <typename T>
__global__ void __launch_bounds__(kST)
scan_down_kernel(const T *__restrict__ in, uint64_t n, const T *__restrict__ offs,
                 T *__restrict__ out, T *__restrict__ total_max) {
    __shared__ T s_warp[kST / 32];
    __shared__ T total;
    const uint64_t t0 = (uint64_t)blockIdx.x * kSTile + (uint64_t)threadIdx.x * kSIPT;
    T v[kSIPT];
    T acc = 0;
#pragma unroll
    for (int j = 0; j < kSIPT; j++) {
        v[j] = (t0 + j < n) ? in[t0 + j] : (T)0;
        acc += v[j];
    }
    T run = block_exscan<T>(acc, s_warp, &total) + (offs ? offs[blockIdx.x] : (T)0);
#pragma unroll
    for (int j = 0; j < kSIPT; j++) {
        if (t0 + j < n) out[t0 + j] = run;
        run += v[j];
    }
    if (total_max) {
        T m = 0;
#pragma unroll
        for (int j = 0; j < kSIPT; j++) m = v[j] > m ? v[j] : m;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const T y = __shfl_xor_sync(0xffffffffu, m, o);
            m = y > m ? y : m;
        }
        if ((threadIdx.x & 31) == 0 && m)
            atomicMax(reinterpret_cast<unsigned long long *>(total_max) + 1, (unsigned long long)m);
        if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
            *total_max = total + (offs ? offs[blockIdx.x] : (T)0);
    }
}

// Scratch elements scan_run needs for n inputs (block sums and offsets of
// every recursion level).
uint64_t scan_ws_elems(uint64_t n) {
    uint64_t total = 0;
    while (n > (uint64_t)kSTile) {
        n = (n + kSTile - 1) / kSTile;
        total += 2 * n;
    }
    return total;
}

// Exclusive scan d_out = scan(d_in) with caller-provided scratch (ws of
// scan_ws_elems(n) elements); d_total (optional, two words) receives the sum
// and the largest input.
template <typename T>
bt_status scan_run(const T *d_in, T *d_out, uint64_t n, T *d_total, T *ws, cudaStream_t s) {
    if (n == 0) {
        if (d_total) BT_CUDA(cudaMemsetAsync(d_total, 0, 2 * sizeof(T), s));
        return BT_OK;
    }
    const uint64_t nb = (n + kSTile - 1) / kSTile;
    if (nb == 1) {
        count_launch();
        scan_down_kernel<T><<<1, kST, 0, s>>>(d_in, n, nullptr, d_out, d_total);
        BT_CUDA(cudaGetLastError());
        return BT_OK;
    }
    T *sums = ws, *offs = ws + nb;
    count_launch();
    scan_reduce_kernel<T><<<(unsigned)nb, kST, 0, s>>>(d_in, n, sums);
    bt_status st = scan_run<T>(sums, offs, nb, nullptr, ws + 2 * nb, s);
    if (st != BT_OK) return st;
    count_launch();
    scan_down_kernel<T><<<(unsigned)nb, kST, 0, s>>>(d_in, n, offs, d_out, d_total);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

template <typename T>
bt_status scan_impl(const T *d_in, T *d_out, uint64_t n, T *d_total, cudaStream_t s) {
    if (d_total) BT_CUDA(cudaMemsetAsync(d_total, 0, 2 * sizeof(T), s));
    const uint64_t we = scan_ws_elems(n);
    T *ws = nullptr;
    if (we) {
        bt_status st = ws_alloc((void **)&ws, we * sizeof(T), s);
        if (st != BT_OK) return st;
    }
    bt_status st = scan_run<T>(d_in, d_out, n, d_total, ws, s);
    ws_free(ws, s);
    return st;
}

// -------------------------------------------------------- partition host --

// One-time raise of a scatter instantiation's dynamic shared memory above the
// 48 KB default (function attributes are per device; the server's worker and
// user threads may partition at once).
template <typename K, typename P, bool HAS_B, bool SORT, typename IO>
bt_status scatter_smem_attr() {
    static std::atomic<bool> done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && done[dev].load(std::memory_order_acquire)) return BT_OK;
    BT_CUDA(cudaFuncSetAttribute(part_scatter_kernel<K, P, HAS_B, SORT, IO>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)PartSmem<K, P, HAS_B>::bytes));
    if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    return BT_OK;
}

// The tables of a pass: a row per chunk and the totals, then a row per tile
// when chunks have several.
size_t part_table_bytes(uint64_t n, uint32_t tile_cap) {
    const uint64_t ntiles = (n + tile_cap - 1) / tile_cap;
    return (size_t)(kPartMaxChunks + 1 + ntiles) * 256 * sizeof(uint32_t);
}

template <typename K, typename P, bool HAS_B, bool SORT, typename IO>
bt_status part_pass(const IO &io, uint64_t n, GroupKeyParams gp, int pass, uint32_t *table,
                    cudaStream_t s) {
    bt_status st = scatter_smem_attr<K, P, HAS_B, SORT, IO>();
    if (st != BT_OK) return st;
    const uint64_t sms = (uint64_t)sm_count();
    const PartCut cut = part_cut(n, PartSmem<K, P, HAS_B>::T, sms);
    uint32_t *tile_tab = cut.per > 1 ? table + (kPartMaxChunks + 1) * 256 : nullptr;
    count_launch();
    part_count_kernel<K, P, HAS_B, SORT, IO><<<cut.nchunks, kPT, 0, s>>>(io, cut, gp, pass, table, tile_tab);
    if (!cut.direct) {
        count_launch();
        part_prefix_kernel<<<32, 256, 0, s>>>(table, (int)cut.nchunks);
    }
    count_launch();
    part_scatter_kernel<K, P, HAS_B, SORT, IO>
        <<<(unsigned)std::min<uint64_t>(cut.ntiles, kPartCtas * sms), kPT, PartSmem<K, P, HAS_B>::bytes, s>>>(
            io, cut, gp, pass, table, tile_tab);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

template <typename K, bool HAS_B>
bt_status partition_impl(const bt_tree *t, int kind, const K *d_a, const K *d_b, uint64_t nq,
                         K *out_a, K *out_b, uint32_t *out_perm, cudaStream_t s) {
    GroupKeyParams gp;
    gp.kind = kind;
    gp.cbits = kind == kPartPoint ? kPointGroupBits : kRangeGroupBits;  // per coordinate
    gp.shift = std::max(0, bitlen64(t->max_key) - gp.cbits);
    const int passes = ((kind == kPartPoint ? 1 : 2) * gp.cbits + 7) / 8;
    if (passes > 2) return fail(BT_ERR_INTERNAL, "partition supports at most two passes");
    // the table and, for two passes, one intermediate copy of the items
    const size_t ab = align256(nq * sizeof(K)), pb = align256(nq * sizeof(uint32_t));
    WsGuard ws(s);
    const size_t tb = align256(part_table_bytes(nq, PartSmem<K, uint32_t, HAS_B>::T));
    bt_status st = ws.alloc(tb + (passes > 1 ? ab * (HAS_B ? 2 : 1) + pb : 0));
    if (st != BT_OK) return st;
    unsigned char *p = ws.as<unsigned char>();
    uint32_t *table = reinterpret_cast<uint32_t *>(p);
    using IO = PassIO<K, uint32_t>;
    IO io{d_a, d_b, nullptr, out_a, out_b, out_perm};
    if (passes > 1) {
        p += tb;
        IO mid = io;
        mid.a_out = reinterpret_cast<K *>(p);
        mid.b_out = HAS_B ? reinterpret_cast<K *>(p + ab) : nullptr;
        mid.p_out = reinterpret_cast<uint32_t *>(p + ab * (HAS_B ? 2 : 1));
        st = part_pass<K, uint32_t, HAS_B, false, IO>(mid, nq, gp, 0, table, s);
        if (st != BT_OK) return st;
        io.a_in = mid.a_out;
        io.b_in = mid.b_out;
        io.p_in = mid.p_out;
    }
    return part_pass<K, uint32_t, HAS_B, false, IO>(io, nq, gp, passes - 1, table, s);
}

// LSD radix sort of n keys carrying a payload (p_in, or the item's index when
// p_in is null): pass p partitions by byte p of the key (stable), so after
// the last pass the keys are sorted and equal keys keep their input order.
// The values travel with their keys: carrying the index and gathering the
// values at the end cost 1.18 ms of random reads at 2^26 u32 pairs, more
// than all passes' extra bytes.
template <typename K, typename P>
bt_status radix_sort(const K *d_keys, const P *p_in, uint64_t n, int passes, K *out_keys, P *out_p,
                     cudaStream_t s) {
    const size_t kb = align256(n * sizeof(K)), pb = align256(n * sizeof(P));
    const size_t tb = align256(part_table_bytes(n, PartSmem<K, P, false>::T));
    WsGuard ws(s);
    bt_status st = ws.alloc(256 + tb + kb + pb);
    if (st != BT_OK) return st;
    unsigned char *w = ws.as<unsigned char>();
    using IO = SortIO<K, P>;
    IO io;
    io.in = d_keys;
    io.p_in = p_in;
    io.out = out_keys;
    io.p_out = out_p;
    io.vary = reinterpret_cast<unsigned long long *>(w);
    io.passes = passes;
    uint32_t *table = reinterpret_cast<uint32_t *>(w + 256);
    io.tk = reinterpret_cast<K *>(w + 256 + tb);
    io.tp = reinterpret_cast<P *>(w + 256 + tb + kb);
    BT_CUDA(cudaMemsetAsync(io.vary, 0, sizeof(*io.vary), s));
    GroupKeyParams gp{kPartRadix, 0, 8};
    for (int p = 0; p < passes && st == BT_OK; p++)
        st = part_pass<K, P, false, true, IO>(io, n, gp, p, table, s);
    return st;
}

bt_status order_u16_impl(const uint32_t *d_keys, uint64_t n, uint32_t *d_perm, cudaStream_t s) {
    WsGuard ws(s);  // the sorted keys, which nobody reads
    bt_status st = ws.alloc(n * sizeof(uint32_t));
    if (st != BT_OK) return st;
    return radix_sort<uint32_t, uint32_t>(d_keys, nullptr, n, 2, ws.as<uint32_t>(), d_perm, s);
}

// Single-pass point partition into caller-provided memory (no allocation):
// the table comes from `ws` (partition_point_ws_bytes bytes).
template <typename K>
bt_status partition_point_prealloc(const bt_tree *t, const K *d_q, uint64_t nq, K *out_q,
                                   uint32_t *out_perm, unsigned char *ws, cudaStream_t s) {
    GroupKeyParams gp;
    gp.kind = kPartPoint;
    gp.cbits = kPointGroupBits;
    gp.shift = std::max(0, bitlen64(t->max_key) - gp.cbits);
    using IO = PassIO<K, uint32_t>;
    return part_pass<K, uint32_t, false, false, IO>(IO{d_q, nullptr, nullptr, out_q, nullptr, out_perm},
                                                    nq, gp, 0, reinterpret_cast<uint32_t *>(ws), s);
}

// --------------------------------------------------------- range fill ----

// One warp per query: ids[off .. off+cnt) = values of positions lb .. lb+cnt
// (read from the leaf blocks, S values per block).  SORT: up to kWarpSortCap
// values are put in ascending order on the way (in registers; a fill and a
// sort of its own read and wrote every ID once more: 2^20 ranges, 34 M IDs,
// 0.169 + 0.220 ms, fused 0.263).  A warp takes `per` consecutive queries at a
// time, so that their counts, bounds and offsets arrive in three loads: 32 in
// large batches, fewer in those that would leave warps idle.  Queries of more
// than kFillLong values are left to the whole CTA, which reads eight values per
// thread at a time.  Whole searches over 2^24 keys with 32 queries to every warp
// and one warp to a query / now: 64 ranges of up to 20,000 values 1.47 / 0.10 ms,
// 16 of up to 10^6 25.3 / 1.25 ms, 4,096 of up to 1,000 0.165 / 0.078 ms.
constexpr int kFillThreads = 256;
constexpr int kFillWarps = kFillThreads / 32;
constexpr uint64_t kFillLong = 2048;

template <typename K, typename V, bool SORT>
__global__ void __launch_bounds__(kFillThreads)
range_fill_kernel(const unsigned char *__restrict__ leaves, const uint64_t *__restrict__ lb,
                  const uint64_t *__restrict__ cnt, const uint64_t *__restrict__ off, uint64_t nq,
                  uint32_t per, V *__restrict__ ids) {
    using LG = LeafGeom<K, V>;
    __shared__ unsigned s_long[kFillWarps];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint64_t step = (uint64_t)kFillWarps * per;  // the CTA's queries of one round
    bool more = false;
    auto value = [&](uint64_t p) {
        return __ldg(reinterpret_cast<const V *>(leaves + (p / LG::S) * LG::BS + kSectorBytes) + p % LG::S);
    };
    for (uint64_t b0 = blockIdx.x * step; b0 < nq; b0 += gridDim.x * step) {
        const uint64_t i = b0 + w * per + lane;
        const bool mine = lane < per && i < nq;
        const uint64_t mc = mine ? cnt[i] : 0, ml = mine ? lb[i] : 0, mo = mine ? off[i] : 0;
        more |= mc > kFillLong;
        unsigned todo = __ballot_sync(0xffffffffu, mc != 0 && mc <= kFillLong);
        while (todo) {
            const int j = __ffs((int)todo) - 1;
            todo &= todo - 1;
            const uint32_t c = __shfl_sync(0xffffffffu, (uint32_t)mc, j);
            const uint64_t l = __shfl_sync(0xffffffffu, ml, j);
            V *dst = ids + __shfl_sync(0xffffffffu, mo, j);
            if (SORT && c > 1 && c <= (uint32_t)kWarpSortCap) {
                auto at = [&](uint32_t e) { return value(l + e); };
                warp_sort_small<V>(at, dst, c, (int)lane);
            } else {
#pragma unroll 4
                for (uint32_t k = lane; k < c; k += 32) dst[k] = value(l + k);
            }
        }
    }
    if (!__syncthreads_or(more)) return;
    for (uint64_t b0 = blockIdx.x * step; b0 < nq; b0 += gridDim.x * step) {
        const uint64_t i = b0 + threadIdx.x;  // step <= kFillThreads
        const bool big = threadIdx.x < step && i < nq && cnt[i] > kFillLong;
        const unsigned m = __ballot_sync(0xffffffffu, big);
        if (lane == 0) s_long[w] = m;
        __syncthreads();
        for (int z = 0; z < kFillWarps; z++) {
            for (unsigned todo = s_long[z]; todo; todo &= todo - 1) {
                const uint64_t j = b0 + z * 32 + __ffs((int)todo) - 1;
                const uint64_t c = cnt[j], l = lb[j];
                V *dst = ids + off[j];
                constexpr int U = 8;
                uint64_t k = threadIdx.x;
                for (; k + (U - 1) * kFillThreads < c; k += U * kFillThreads) {
                    V v[U];
#pragma unroll
                    for (int u = 0; u < U; u++) v[u] = value(l + k + u * kFillThreads);
#pragma unroll
                    for (int u = 0; u < U; u++) dst[k + u * kFillThreads] = v[u];
                }
                for (; k < c; k += kFillThreads) dst[k] = value(l + k);
            }
        }
        __syncthreads();
    }
}

// Sorts each query's ID segment when values do not ascend with keys.  Up to
// kWarpSortCap values: sorted by the pass that wrote them, one warp in
// registers (warp_sort_small, a bitonic network).  Up to kWarpLongCap: the
// same, by a pass of its own over the listed segments.  Up to kSortBytes of
// values: one CTA per segment, bitonic network in shared memory.  Longer: one
// CTA each by a bitonic network over a padded copy in global memory.
constexpr int kWarpLongCap = 1024;
constexpr size_t kSortBytes = 128 * 1024;
constexpr unsigned int kMedListCap = 1u << 16;

// Lists the segments of kWarpSortCap < c <= cap (*n_med of them, the first
// kMedListCap in med_list).
__global__ void __launch_bounds__(256)
list_med_segments(const uint64_t *__restrict__ cnt, uint64_t nq, uint64_t cap,
                  unsigned int *__restrict__ n_med, uint64_t *__restrict__ med_list) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nq;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t c = cnt[i];
        if (c > (uint64_t)kWarpSortCap && c <= cap) {
            const unsigned int k = atomicAdd(n_med, 1u);
            if (k < kMedListCap) med_list[k] = i;
        }
    }
}

// One warp per listed segment of up to kWarpLongCap values (every segment
// when the list overflowed).  A CTA per segment, its network in shared memory
// with a barrier per step, took 0.43 ms for some
// 14,000 segments of 257 to 400 values; this takes 0.058.
template <typename V>
__global__ void __launch_bounds__(128)
warp_long_sort_kernel(const uint64_t *__restrict__ cnt, const uint64_t *__restrict__ off, uint64_t nq,
                      const unsigned int *__restrict__ n_med, const uint64_t *__restrict__ med_list,
                      V *__restrict__ ids) {
    const int lane = threadIdx.x & 31;
    const unsigned int nm = *n_med;
    const bool listed = nm <= kMedListCap;
    const uint64_t n = listed ? nm : nq;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t k = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; k < n; k += nw) {
        const uint64_t i = listed ? med_list[k] : k;
        const uint64_t c = cnt[i];
        if (c <= (uint64_t)kWarpSortCap || c > (uint64_t)kWarpLongCap) continue;
        V *seg = ids + off[i];
        auto at = [&](uint32_t e) { return seg[e]; };
        if (c <= 512) warp_sort_copy<V, 16>(at, seg, (uint32_t)c, lane);
        else warp_sort_copy<V, 32>(at, seg, (uint32_t)c, lane);
    }
}

// One CTA per segment of kWarpLongCap < c <= cap: the listed ones, or every
// one when the list overflowed.  Shared memory for the next power of two of
// the largest.
template <typename V>
__global__ void __launch_bounds__(512)
segment_sort_kernel(const uint64_t *__restrict__ cnt, const uint64_t *__restrict__ off, uint64_t nq,
                    uint64_t cap, const unsigned int *__restrict__ n_med,
                    const uint64_t *__restrict__ list, V *__restrict__ ids) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *buf = reinterpret_cast<V *>(smem_raw);
    const unsigned int nm = *n_med;
    const bool listed = nm <= kMedListCap;
    const uint64_t n = listed ? nm : nq;
    for (uint64_t li = blockIdx.x; li < n; li += gridDim.x) {
        const uint64_t i = listed ? list[li] : li;
        const uint64_t c = cnt[i];
        if (c <= (uint64_t)kWarpLongCap || c > cap) continue;
        uint32_t p2 = 1;
        while (p2 < c) p2 <<= 1;
        V *seg = ids + off[i];
        for (uint32_t k = threadIdx.x; k < p2; k += blockDim.x) buf[k] = k < c ? seg[k] : key_max<V>();
        __syncthreads();
        for (uint32_t size = 2; size <= p2; size <<= 1) {
            for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
                // pair z: slots k and k + stride
                for (uint32_t z = threadIdx.x; z < p2 / 2; z += blockDim.x) {
                    const uint32_t k = ((z & ~(stride - 1)) << 1) | (z & (stride - 1));
                    const V x = buf[k], y = buf[k + stride];
                    if ((x > y) == ((k & size) == 0)) {
                        buf[k] = y;
                        buf[k + stride] = x;
                    }
                }
                __syncthreads();
            }
        }
        for (uint32_t k = threadIdx.x; k < c; k += blockDim.x) seg[k] = buf[k];
        __syncthreads();
    }
}

// Segments longer than cap: list them (offset, count).
__global__ void list_long_segments(const uint64_t *__restrict__ cnt, const uint64_t *__restrict__ off,
                                   uint64_t nq, uint64_t cap, unsigned int *__restrict__ n_long,
                                   uint64_t *__restrict__ list, unsigned int max_list) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nq;
         i += (uint64_t)gridDim.x * blockDim.x) {
        if (cnt[i] > cap) {
            const unsigned int k = atomicAdd(n_long, 1u);
            if (k < max_list) {
                list[2 * k] = off[i];
                list[2 * k + 1] = cnt[i];
            }
        }
    }
}

// One CTA sorts one long segment: copy into a power-of-two scratch padded
// with all-ones, bitonic network in global (L2-resident) memory, copy back.
template <typename V>
__global__ void __launch_bounds__(1024)
long_segment_sort(V *__restrict__ ids, uint64_t off, uint64_t c, V *__restrict__ tmp, uint64_t p2) {
    for (uint64_t k = threadIdx.x; k < p2; k += blockDim.x) tmp[k] = k < c ? ids[off + k] : key_max<V>();
    __syncthreads();
    for (uint64_t size = 2; size <= p2; size <<= 1) {
        for (uint64_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint64_t k = threadIdx.x; k < p2; k += blockDim.x) {
                const uint64_t partner = k ^ stride;
                if (partner > k) {
                    const bool asc = (k & size) == 0;
                    const V x = tmp[k], y = tmp[partner];
                    if ((x > y) == asc) {
                        tmp[k] = y;
                        tmp[partner] = x;
                    }
                }
            }
            __syncthreads();
        }
    }
    for (uint64_t k = threadIdx.x; k < c; k += blockDim.x) ids[off + k] = tmp[k];
}

}  // namespace

bt_status launch_partition(const bt_tree *t, int kind, const void *d_a, const void *d_b,
                           uint64_t nq, void *d_out_a, void *d_out_b, uint32_t *d_perm,
                           cudaStream_t s) {
    if (nq == 0) return BT_OK;
    if (nq >= (1ull << 32)) return fail(BT_ERR_INVALID_ARGUMENT, "grouped batches need nq < 2^32");
    const bool hb = kind != kPartPoint;
    if (t->key_bytes == 4)
        return hb ? partition_impl<uint32_t, true>(t, kind, (const uint32_t *)d_a,
                                                   (const uint32_t *)d_b, nq, (uint32_t *)d_out_a,
                                                   (uint32_t *)d_out_b, d_perm, s)
                  : partition_impl<uint32_t, false>(t, kind, (const uint32_t *)d_a, nullptr, nq,
                                                    (uint32_t *)d_out_a, nullptr, d_perm, s);
    return hb ? partition_impl<uint64_t, true>(t, kind, (const uint64_t *)d_a,
                                               (const uint64_t *)d_b, nq, (uint64_t *)d_out_a,
                                               (uint64_t *)d_out_b, d_perm, s)
              : partition_impl<uint64_t, false>(t, kind, (const uint64_t *)d_a, nullptr, nq,
                                                (uint64_t *)d_out_a, nullptr, d_perm, s);
}

bt_status launch_sort_pairs(int key_bytes, int value_bytes, const void *d_keys, const void *d_vals,
                            uint64_t n, void *out_keys, void *out_vals, cudaStream_t s) {
    if (n == 0) return BT_OK;
    if (n >= (1ull << 32)) return fail(BT_ERR_INVALID_ARGUMENT, "sort needs fewer than 2^32 pairs");
    if (key_bytes == 4)
        return value_bytes == 4
                   ? radix_sort<uint32_t, uint32_t>((const uint32_t *)d_keys, (const uint32_t *)d_vals, n, 4,
                                                         (uint32_t *)out_keys, (uint32_t *)out_vals, s)
                   : radix_sort<uint32_t, uint64_t>((const uint32_t *)d_keys, (const uint64_t *)d_vals, n, 4,
                                                         (uint32_t *)out_keys, (uint64_t *)out_vals, s);
    return value_bytes == 4
               ? radix_sort<uint64_t, uint32_t>((const uint64_t *)d_keys, (const uint32_t *)d_vals, n, 8,
                                                     (uint64_t *)out_keys, (uint32_t *)out_vals, s)
               : radix_sort<uint64_t, uint64_t>((const uint64_t *)d_keys, (const uint64_t *)d_vals, n, 8,
                                                     (uint64_t *)out_keys, (uint64_t *)out_vals, s);
}

bt_status launch_order_u16(const uint32_t *d_keys, uint64_t n, uint32_t *d_perm, cudaStream_t s) {
    if (n == 0) return BT_OK;
    if (n >= (1ull << 32)) return fail(BT_ERR_INVALID_ARGUMENT, "ordering needs n < 2^32");
    return order_u16_impl(d_keys, n, d_perm, s);
}

size_t partition_point_ws_bytes(uint64_t nq) {
    return std::max(part_table_bytes(nq, PartSmem<uint32_t, uint32_t, false>::T),
                    part_table_bytes(nq, PartSmem<uint64_t, uint32_t, false>::T));
}

bt_status launch_partition_point_prealloc(const bt_tree *t, const void *d_q, uint64_t nq,
                                          void *out_q, uint32_t *out_perm, void *ws,
                                          cudaStream_t s) {
    if (nq == 0) return BT_OK;
    if (t->key_bytes == 4)
        return partition_point_prealloc<uint32_t>(t, (const uint32_t *)d_q, nq, (uint32_t *)out_q,
                                                  out_perm, (unsigned char *)ws, s);
    return partition_point_prealloc<uint64_t>(t, (const uint64_t *)d_q, nq, (uint64_t *)out_q,
                                              out_perm, (unsigned char *)ws, s);
}

bt_status launch_scan_u64(const uint64_t *d_in, uint64_t *d_out, uint64_t n, uint64_t *d_total,
                          cudaStream_t s) {
    return scan_impl<uint64_t>(d_in, d_out, n, d_total, s);
}

namespace {
template <typename K, typename B>
bt_status bucket_impl(const bt_tree *t, const BucketMap &map, const B &q, uint64_t nq, K *out_q,
                      uint32_t *pos, const BucketPlan &bp, cudaStream_t s) {
    static std::atomic<bool> done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_acquire)) {
        BT_CUDA(cudaFuncSetAttribute(bucket_scatter_kernel<K, B>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)BucketSmem<K>::bytes));
        if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    }
    uint32_t *total = bp.scratch, *cursor = bp.scratch + kMaxBuckets;
    BT_CUDA(cudaMemsetAsync(total, 0, kMaxBuckets * sizeof(uint32_t), s));
    const uint64_t sms = (uint64_t)sm_count();
    count_launch();
    bucket_count_kernel<K, B><<<(unsigned)std::min<uint64_t>((nq + kBT * 8 - 1) / (kBT * 8), sms * 4), kBT, 0, s>>>(
        q, nq, map, total);
    count_launch();
    bucket_start_kernel<K><<<1 + ((map.last + 2) * 8 + 1023) / 1024, 1024, 0, s>>>(
        t->dev, map, bucket_slice(nq), total, cursor, bp.first, bp.items, bp.n_items);
    count_launch();
    constexpr uint64_t T = BucketSmem<K>::T;
    bucket_scatter_kernel<K, B><<<(unsigned)std::min<uint64_t>((nq + T - 1) / T, sms * 2), kBT,
                                  BucketSmem<K>::bytes, s>>>(q, nq, map, cursor, out_q, pos);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

template <typename K>
bt_status bucket_k(const bt_tree *t, const BucketMap &map, const void *d_q, const void *d_hi,
                   uint64_t nq, void *out_q, uint32_t *pos, const BucketPlan &bp, cudaStream_t s) {
    if (!d_hi)
        return bucket_impl<K>(t, map, PointBatch<K>{(const K *)d_q}, nq, (K *)out_q, pos, bp, s);
    return bucket_impl<K>(t, map, RangeBatch<K>{(const K *)d_q, (const K *)d_hi, nq}, 2 * nq,
                          (K *)out_q, pos, bp, s);
}
}  // namespace

bt_status launch_buckets(const bt_tree *t, const BucketMap &map, const void *d_q, const void *d_hi,
                         uint64_t nq, void *out_q, uint32_t *pos, const BucketPlan &bp,
                         cudaStream_t s) {
    return t->key_bytes == 4 ? bucket_k<uint32_t>(t, map, d_q, d_hi, nq, out_q, pos, bp, s)
                             : bucket_k<uint64_t>(t, map, d_q, d_hi, nq, out_q, pos, bp, s);
}

bt_status launch_range_gather(const bt_tree *t, const uint32_t *rank, const uint32_t *pos,
                              const void *d_lo, const void *d_hi, uint64_t nr, uint64_t *d_counts,
                              uint64_t *d_lb, cudaStream_t s) {
    const unsigned grid = (unsigned)((nr + 2047) / 2048);
    count_launch();
    if (t->key_bytes == 4)
        range_gather_kernel<uint32_t><<<grid, 512, 0, s>>>(rank, pos, (const uint32_t *)d_lo,
                                                           (const uint32_t *)d_hi, nr,
                                                           (uint32_t)t->max_key, t->n, d_counts, d_lb);
    else
        range_gather_kernel<uint64_t><<<grid, 512, 0, s>>>(rank, pos, (const uint64_t *)d_lo,
                                                           (const uint64_t *)d_hi, nr, t->max_key,
                                                           t->n, d_counts, d_lb);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

bt_status launch_bucket_blocks(const bt_tree *t, const unsigned int *d_unsorted, uint32_t *d_blocks,
                               cudaStream_t s) {
    const unsigned grid = kMaxBuckets * 8 / 256;
    const unsigned char *lv = (const unsigned char *)t->d_leaves;
    const uint64_t S = kSectorBytes / t->key_bytes;
    const unsigned char *last = lv + (t->n - 1) / S * leaf_stride(t->key_bytes, t->val_bytes) +
                                (t->n - 1) % S * t->key_bytes;
    count_launch();
    if (t->key_bytes == 4)
        bucket_blocks_kernel<uint32_t><<<grid, 256, 0, s>>>(t->dev, (const uint32_t *)lv,
                                                            (const uint32_t *)last, d_unsorted, d_blocks);
    else
        bucket_blocks_kernel<uint64_t><<<grid, 256, 0, s>>>(t->dev, (const uint64_t *)lv,
                                                            (const uint64_t *)last, d_unsorted, d_blocks);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

bt_status launch_bucket_gather(int val_bytes, const void *res, const uint8_t *rfound,
                               const uint32_t *pos, uint64_t nq, void *d_out, uint8_t *d_found,
                               cudaStream_t s) {
    const unsigned grid = (unsigned)((nq + 4095) / 4096);
    count_launch();
    if (val_bytes == 4)
        bucket_gather_kernel<uint32_t><<<grid, 512, 0, s>>>((const uint32_t *)res, rfound, pos, nq,
                                                            (uint32_t *)d_out, d_found);
    else
        bucket_gather_kernel<uint64_t><<<grid, 512, 0, s>>>((const uint64_t *)res, rfound, pos, nq,
                                                            (uint64_t *)d_out, d_found);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

namespace {
template <typename K, typename V>
void range_fill(const bt_tree *t, const uint64_t *d_lb, const uint64_t *d_counts,
                const uint64_t *d_offsets, uint64_t nq, V *ids, cudaStream_t s) {
    const uint64_t ctas = (uint64_t)sm_count() * 8;
    const uint32_t per = (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(1, nq / (ctas * kFillWarps)));
    const uint64_t step = (uint64_t)kFillWarps * per;
    const unsigned grid = (unsigned)std::min<uint64_t>((nq + step - 1) / step, ctas);
    const unsigned char *lv = (const unsigned char *)t->d_leaves;
    if (t->values_sorted)
        range_fill_kernel<K, V, false><<<grid, kFillThreads, 0, s>>>(lv, d_lb, d_counts, d_offsets, nq, per, ids);
    else
        range_fill_kernel<K, V, true><<<grid, kFillThreads, 0, s>>>(lv, d_lb, d_counts, d_offsets, nq, per, ids);
}
}  // namespace

bt_status launch_range_fill(const bt_tree *t, const uint64_t *d_lb, const uint64_t *d_counts,
                            const uint64_t *d_offsets, uint64_t nq, uint64_t max_count, void *d_ids,
                            cudaStream_t s) {
    if (nq == 0 || t->n == 0) return BT_OK;
    count_launch();
    if (t->key_bytes == 4 && t->val_bytes == 4)
        range_fill<uint32_t, uint32_t>(t, d_lb, d_counts, d_offsets, nq, (uint32_t *)d_ids, s);
    else if (t->key_bytes == 4)
        range_fill<uint32_t, uint64_t>(t, d_lb, d_counts, d_offsets, nq, (uint64_t *)d_ids, s);
    else if (t->val_bytes == 4)
        range_fill<uint64_t, uint32_t>(t, d_lb, d_counts, d_offsets, nq, (uint32_t *)d_ids, s);
    else
        range_fill<uint64_t, uint64_t>(t, d_lb, d_counts, d_offsets, nq, (uint64_t *)d_ids, s);
    BT_CUDA(cudaGetLastError());
    if (t->values_sorted) return BT_OK;
    return launch_segment_sort(t, d_counts, d_offsets, nq, max_count, d_ids, s);
}

bt_status launch_segment_sort(const bt_tree *t, const uint64_t *d_counts, const uint64_t *d_offsets,
                              uint64_t nq, uint64_t max_count, void *d_ids, cudaStream_t s) {
    if (nq == 0 || max_count <= (uint64_t)kWarpSortCap) return BT_OK;
    WsGuard g_stat(s), g_med(s);
    bt_status st = g_stat.alloc(sizeof(unsigned int));
    if (st == BT_OK) st = g_med.alloc(kMedListCap * sizeof(uint64_t));
    if (st != BT_OK) return st;
    unsigned int *stat = g_stat.as<unsigned int>();
    uint64_t *med = g_med.as<uint64_t>();
    BT_CUDA(cudaMemsetAsync(stat, 0, sizeof(unsigned int), s));
    const unsigned sms = (unsigned)sm_count();
    const uint64_t cap = kSortBytes / (uint64_t)t->val_bytes;
    count_launch();
    list_med_segments<<<(unsigned)std::min<uint64_t>((nq + 255) / 256, sms * 8), 256, 0, s>>>(
        d_counts, nq, cap, stat, med);
    count_launch();
    if (t->val_bytes == 4)
        warp_long_sort_kernel<uint32_t><<<sms * 4, 128, 0, s>>>(d_counts, d_offsets, nq, stat, med,
                                                                (uint32_t *)d_ids);
    else
        warp_long_sort_kernel<uint64_t><<<sms * 4, 128, 0, s>>>(d_counts, d_offsets, nq, stat, med,
                                                                (uint64_t *)d_ids);
    BT_CUDA(cudaGetLastError());
    if (max_count > (uint64_t)kWarpLongCap) {
        uint64_t p2 = 2 * kWarpLongCap;
        while (p2 < std::min(max_count, cap)) p2 <<= 1;
        const size_t smem = p2 * (size_t)t->val_bytes;
        const unsigned grid = sms * (unsigned)std::min<size_t>(4, 200 * 1024 / smem);
        count_launch();
        if (t->val_bytes == 4) {
            BT_CUDA(cudaFuncSetAttribute(segment_sort_kernel<uint32_t>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSortBytes));
            segment_sort_kernel<uint32_t><<<grid, 512, smem, s>>>(d_counts, d_offsets, nq, cap, stat, med,
                                                                  (uint32_t *)d_ids);
        } else {
            BT_CUDA(cudaFuncSetAttribute(segment_sort_kernel<uint64_t>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSortBytes));
            segment_sort_kernel<uint64_t><<<grid, 512, smem, s>>>(d_counts, d_offsets, nq, cap, stat, med,
                                                                  (uint64_t *)d_ids);
        }
        BT_CUDA(cudaGetLastError());
    }
    if (max_count <= cap) return BT_OK;
    // some segments exceed the shared-memory sort: list and sort them one CTA each
    const unsigned int max_list = 1u << 16;
    WsGuard g_list(s);
    st = g_list.alloc(2 * (size_t)max_list * sizeof(uint64_t));
    if (st != BT_OK) return st;
    unsigned int *flag = stat;
    uint64_t *d_list = g_list.as<uint64_t>();
    BT_CUDA(cudaMemsetAsync(flag, 0, sizeof(unsigned int), s));
    count_launch();
    list_long_segments<<<(unsigned)std::min<uint64_t>((nq + 255) / 256, 4096), 256, 0, s>>>(
        d_counts, d_offsets, nq, cap, flag, d_list, max_list);
    unsigned int n_long = 0;
    BT_CUDA(cudaMemcpyAsync(&n_long, flag, sizeof(n_long), cudaMemcpyDeviceToHost, s));
    BT_CUDA(cudaStreamSynchronize(s));
    if (n_long > max_list)
        return fail(BT_ERR_NOT_SUPPORTED, "more than 65536 result sets exceed 128 KiB of unsorted values");
    std::vector<uint64_t> list(2 * (size_t)n_long);
    BT_CUDA(cudaMemcpyAsync(list.data(), d_list, list.size() * sizeof(uint64_t),
                            cudaMemcpyDeviceToHost, s));
    BT_CUDA(cudaStreamSynchronize(s));
    const size_t vb = (size_t)t->val_bytes;
    for (unsigned int k = 0; k < n_long && st == BT_OK; k++) {
        const uint64_t off = list[2 * k], c = list[2 * k + 1];
        uint64_t p2 = 1;
        while (p2 < c) p2 <<= 1;
        WsGuard g_tmp(s);
        st = g_tmp.alloc(p2 * vb);
        if (st != BT_OK) break;
        count_launch();
        if (vb == 4)
            long_segment_sort<uint32_t><<<1, 1024, 0, s>>>((uint32_t *)d_ids, off, c, g_tmp.as<uint32_t>(), p2);
        else
            long_segment_sort<uint64_t><<<1, 1024, 0, s>>>((uint64_t *)d_ids, off, c, g_tmp.as<uint64_t>(), p2);
    }
    BT_CUDA(cudaGetLastError());
    return st;
}

}  // namespace bt

extern "C" {

// No partition pass waits on another CTA.
uint64_t bt_partition_lookback_timeouts(void) { return 0; }

}  // extern "C"
