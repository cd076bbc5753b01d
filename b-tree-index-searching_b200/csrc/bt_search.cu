// Point search and range-bound kernels.
//
// point_kernel replaces kernelSearchingNaiveOneStep
// (BPTreeExactSearch.cu:25-105) and, with PERM, the grouped
// kernelSearchingKeyGroupTwoStep (:207-294): same answer (value at the exact
// match, all-ones otherwise), but the grouped variant compares keys, not
// data[] (:269-276), and writes results back in the caller's order.
//
// bounds_line_kernel replaces the range endpoint + count kernels
// (BtreeRangeSearch.cu:215-374 and :33-211).  With implicit leaf positions
// the count is upper_bound(hi) - lower_bound(lo); no leaf-chain walk.
//
// Both kernels are persistent (grid = SMs x resident CTAs), stage one
// separator level into shared memory once per CTA, then loop over warp tiles
// of 32 queries (see bt_search.cuh for the two-phase descent).
// A point query's leaf block -- key sector and value sector side by side, one
// 64-byte DRAM access -- is read by one thread or a lane pair (leaf_answers),
// so a hit costs one HBM round trip.  2^20 u32 keys, 2^20 queries (in L2):
// 36 -> 25.8 us a call against four lanes per query, 34.9 -> 23.5 with the padded
// window and two CTAs per SM; what is left is the instruction
// issue of the shared-memory search and of the one separator line below it.
#include <map>
#include <mutex>
#include <type_traits>

#include "bt_search.cuh"

namespace bt {

// Lanes per query (G) below the staged level and rounds (R) per warp tile of
// 32 queries; each group keeps G/R queries in flight.  Set per tree by
// bt_set_search_config / the autotuner.
struct SearchCfg {
    int g, r;
};
constexpr SearchCfg kSearchCfgs[] = {{8, 1}, {8, 2}, {4, 1}, {4, 2}, {2, 1}};
constexpr int kNumSearchCfgs = sizeof(kSearchCfgs) / sizeof(kSearchCfgs[0]);

int search_cfg_index(int g, int r) {
    for (int k = 0; k < kNumSearchCfgs; k++)
        if (kSearchCfgs[k].g == g && kSearchCfgs[k].r == r) return k;
    return -1;
}

int search_cfg_lanes(int cfg) { return kSearchCfgs[cfg].g; }
int search_cfg_rounds(int cfg) { return kSearchCfgs[cfg].r; }

// The shapes of a tree nobody has set one for (us; 2^19 queries or ranges):
//                          (2,1)  (4,1)  (4,2)  (8,1)  (8,2)
//   point u32, 2^20 keys                 (4,1) fastest throughout
//   point u64, 2^20 keys    46.0   31.3   30.8   27.3   25.2
//   point u64, 2^28         82.7   52.1   54.0   46.5   47.7
//   range u32, 2^20 / 2^26  32/46  48/64  36/49  98/139 63/85
//   range u64, 2^20 / 2^26  74/105 73/104 59/82  144/189 93/124
// A batch of a few warps waits for one chain of reads, which two rounds make
// longer: u64 keys, 2^26, 64 queries: (4,1) 19.1 (8,2) 21.1; 64 ranges: (2,1) 24.2
// (4,2) 28.7, 2^16 ranges 30.9 / 34.5, 2^17 42.8 / 40.8.
int own_search_cfg(int key_bytes, int op, uint64_t nq) {
    if (op == BT_OP_RANGE)
        return key_bytes == 4 || nq < (1ull << 17) ? search_cfg_index(2, 1) : search_cfg_index(4, 2);
    return key_bytes == 4 || nq < 512 ? search_cfg_index(4, 1) : search_cfg_index(8, 2);
}

static int shape_of(const bt_tree *t, int op, uint64_t nq) {
    return t->search_cfg[op] >= 0 ? t->search_cfg[op] : own_search_cfg(t->key_bytes, op, nq);
}

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;

// Shared memory of a search CTA: the staged level, then (bounds kernel) 64
// 8-byte results per warp.
__host__ __device__ inline size_t scratch_offset(const DevTree &t) { return ((size_t)t.smem_bytes + 15) / 16 * 16; }

template <typename K, typename V, int G, int R, bool PERM, bool PAIR>
__global__ void __launch_bounds__(kThreads, 2)
point_kernel(const __grid_constant__ DevTree t, const K *__restrict__ q,
             const uint32_t *__restrict__ perm, uint64_t nq, V *__restrict__ out,
             uint8_t *__restrict__ found) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *s_lvl = reinterpret_cast<K *>(smem_raw);
    {
        const K *src = static_cast<const K *>(t.seps) + t.lvl_off[t.smem_level];
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < t.smem_entries; i += kThreads) s_lvl[win_slot(i)] = src[i];
    }
    __syncthreads();

    constexpr int U = 1;  // queries per lane at a time (2: no faster, 1.05x slower on small batches)
    const int lane = threadIdx.x & 31;
    const K tmax = (K)t.max_key;
    const unsigned char *leaves = static_cast<const unsigned char *>(t.leaves);
    // Grouped input (PERM): each CTA takes one contiguous run of warp tiles,
    // so a CTA works one key range and its warps share node lines in L1.
    // Ungrouped input: warp tiles are strided over the whole grid.
    const uint64_t ntiles = (nq + 32 * U - 1) / (32 * U);
    const uint64_t per_cta = PERM ? (ntiles + gridDim.x - 1) / gridDim.x : 0;
    const uint64_t t_begin = PERM ? blockIdx.x * per_cta + (threadIdx.x >> 5)
                                  : (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t t_end = PERM ? min(ntiles, (blockIdx.x + 1) * per_cta) : ntiles;
    const uint64_t t_step = PERM ? (blockDim.x >> 5) : ((uint64_t)gridDim.x * blockDim.x) >> 5;

    for (uint64_t tile = t_begin; tile < t_end; tile += t_step) {
        const uint64_t base = tile * (32 * U);
        K qv[U], qe[U];
        uint32_t node[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint64_t i = base + u * 32 + lane;
            qv[u] = i < nq ? q[i] : (K)0;
            qe[u] = qv[u] < tmax ? qv[u] : tmax;
        }
        win_bound<K, U>(s_lvl, t.smem_entries, qe, node);
#pragma unroll
        for (int u = 0; u < U; u++) node[u] = walk_lanes<K, G, R>(t, t.smem_level + 1, qe[u], node[u], lane);
        leaf_answers<K, V, U, PAIR>(leaves, node, qv, tmax, [&](int u, int l, V v, bool hit) {
            const uint64_t i = base + u * 32 + l;
            if (i >= nq) return;
            const uint64_t d = PERM ? (uint64_t)perm[i] : i;
            out[d] = v;
            if (found) found[d] = hit ? 1 : 0;
        });
    }
}

// Point search over radix-grouped input (the queries ordered by their top
// kPointGroupBits bits below the tree's key length, as bt_group_queries
// leaves them).  One CTA per SM
// takes a contiguous run of the grouped batch.  For the group of its current
// queries it stages in shared memory the group's window of the deepest
// separator level whose window fits (for 2^26 u32 keys and 256 groups: the
// 32,768 leaf-block maxima of the bottom level, 128 KB), so that one binary
// search in shared memory takes a query straight to its leaf block: the only
// global access left is the leaf block itself.  The window of a group [lo,
// hi] is the level's entries from the lower bound of lo to the lower bound
// of hi; every query of the group has its lower bound inside it.  Warps whose
// tile holds a query of another group (tiles at group boundaries, or input
// that is not grouped at all) take the full descent from the root instead,
// so results never depend on the order of the input.
// The group of a key as the grouping pass forms it: its bits above `shift`
// (the tree's key length less kPointGroupBits), the last group taking
// everything above.
constexpr uint64_t kLastGroup = (1u << kPointGroupBits) - 1u;
__device__ __forceinline__ uint64_t group_of(uint64_t k, int shift) {
    const uint64_t g = k >> shift;
    return g < kLastGroup ? g : kLastGroup;
}

constexpr int kWinThreads = 1024;
constexpr int kWinWarps = kWinThreads / 32;
constexpr size_t kWinBytes = 192 * 1024;
// Below this batch size a window staged per CTA costs more than it saves.
constexpr uint64_t kWinMinQueries = 1ull << 21;

template <typename K, typename V, int G, int R>
__global__ void __launch_bounds__(kWinThreads, 1)
point_window_kernel(const __grid_constant__ DevTree t, const K *__restrict__ q,
                    const uint32_t *__restrict__ perm, uint64_t nq, V *__restrict__ out,
                    uint8_t *__restrict__ found, int shift) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *s_win = reinterpret_cast<K *>(smem_raw);
    __shared__ uint32_t s_blk[2];
    constexpr uint32_t kCap = (uint32_t)(kWinBytes / sizeof(K));
    constexpr int F = kLineBytes / (int)sizeof(K);
    constexpr int LOGF = F == 32 ? 5 : 4;
    constexpr uint32_t ROW = sizeof(K) == 4 ? 32u : 16u;  // swizzle row (elements)
    constexpr int NG = 32 / G;
    constexpr int I = G / R;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int grp = lane / G;
    const int gl = lane % G;
    const K tmax = (K)t.max_key;
    const unsigned char *leaves = static_cast<const unsigned char *>(t.leaves);
    const K *seps = static_cast<const K *>(t.seps);
    const uint64_t ntiles = (nq + 31) / 32;
    const uint64_t per_cta = (ntiles + gridDim.x - 1) / gridDim.x;
    const uint64_t c_begin = blockIdx.x * per_cta;
    const uint64_t c_end = min(ntiles, c_begin + per_cta);
    uint64_t staged = ~0ull;  // group whose window is staged (same in every thread)
    int wlvl = 0;
    uint32_t w0 = 0, wm = 1;
    for (uint64_t t0 = c_begin; t0 < c_end; t0 += kWinWarps) {
        const uint64_t b = group_of((uint64_t)q[t0 * 32], shift);  // group of this step's first query
        if (b != staged) {
            __syncthreads();  // the old window is no longer read
            if (threadIdx.x < 2) {
                const uint64_t lo = b << shift;
                const uint64_t hi = b == kLastGroup ? ~0ull : lo | ((1ull << shift) - 1ull);
                const uint64_t k = threadIdx.x == 0 ? lo : hi;
                s_blk[threadIdx.x] = block_lower_bound<K>(t, k < (uint64_t)tmax ? (K)k : tmax);
            }
            __syncthreads();
            // deepest level whose window fits (level 0 holds at most F entries)
            const uint32_t blo = s_blk[0], bhi = s_blk[1];
            wlvl = t.nlevels - 1;
            int sh = 0;
            while (wlvl > 0 && (bhi >> sh) - (blo >> sh) + 1u > kCap) {
                wlvl--;
                sh += LOGF;
            }
            w0 = blo >> sh;
            wm = (bhi >> sh) - w0 + 1u;
            const K *src = seps + t.lvl_off[wlvl] + w0;
            const uint32_t staged_n = (wm + ROW - 1) / ROW * ROW;
            for (uint32_t i = threadIdx.x; i < staged_n; i += blockDim.x)
                s_win[swz<K>(i)] = i < wm ? src[i] : key_max<K>();
            __syncthreads();
            staged = b;
        }
        const uint64_t tile = t0 + warp;
        if (tile >= c_end) continue;
        const uint64_t base = tile * 32;
        const uint64_t my = base + lane;
        const K myq = my < nq ? q[my] : (K)0;
        const uint32_t myperm = my < nq ? perm[my] : 0u;  // loaded early, off the critical path
        const K myqe = myq < tmax ? myq : tmax;
        // phase 1: the window, or (whole warp) the descent from the root
        const bool inwin = my >= nq || group_of((uint64_t)myq, shift) == staged;
        const bool win = __all_sync(0xffffffffu, inwin);
        uint32_t mynode = 0;
        if (win) {
            const uint32_t p = smem_bound<K>(s_win, wm, myqe, false);
            mynode = w0 + (p < wm ? p : wm - 1u);
        }
        const int from = win ? wlvl + 1 : 0;
#pragma unroll
        for (int r = 0; r < R; r++) {
            K qv[I], qe[I];
            bool up[I];
            uint32_t node[I], pv[I];
#pragma unroll
            for (int s = 0; s < I; s++) {
                const int k = r * (NG * I) + s * NG + grp;
                qv[s] = __shfl_sync(0xffffffffu, myq, k);
                node[s] = __shfl_sync(0xffffffffu, mynode, k);
                pv[s] = __shfl_sync(0xffffffffu, myperm, k);
                qe[s] = qv[s] < tmax ? qv[s] : tmax;
                up[s] = false;
            }
            walk_from<K, G, I>(t, from, qe, up, node, grp, gl);
            leaf_point<K, V, G, I>(
                leaves, node, qv, qe, tmax, grp, gl,
                [&](int s) -> V * {
                    const uint64_t qi = base + (uint64_t)(r * (NG * I) + s * NG + grp);
                    if (qi >= nq) return nullptr;
                    return out + pv[s];
                },
                [&](int s) -> uint8_t * { return found ? found + pv[s] : nullptr; });
        }
    }
}

// ---- point search of a batch ordered by bucket (launch_buckets) ------------
//
// A CTA takes one work item: up to bucket_slice queries of one bucket, whose
// leaf blocks lie between first[bucket] and first[bucket + 1].  It stages that
// window of the deepest separator level that fits in its shared memory, 64-bit
// separators as 32-bit offsets where their span allows it, so that one binary
// search there takes a query past every level above -- for most trees straight
// to its leaf block.  Leaf blocks are then read
//   4-byte keys: by a thread per query, four queries at a time: one 32-byte
//     load of the block's keys, then the matching value;
//   8-byte keys: by a lane pair per query, two queries at a time: one lane the
//     key sector, one the value sector, as one request.
// A quarter of the instructions of the lane-quad form of point_kernel (19 a
// query, which bound this kernel to 0.37 ms at 2^26 u32 keys and 2^24
// queries): 0.178 ms with a thread per query, 0.21 with pairs.  With u64 keys
// (2^28, 2^24 queries) the leaf reads' DRAM access rate bounds it: pairs
// 0.56 ms, thread per query 0.60.


constexpr size_t kBktWinBytes = 200 * 1024;
constexpr size_t kBktWinMin = 16 * 1024;  // room for some level of any tree

// What a bucket search writes: values, or (BOUND) ranks of lower bounds.
template <typename V, bool BOUND>
using BktOut = std::conditional_t<BOUND, uint32_t, V>;

// The qn queries of an item by their staged window: node = w0 + position in
// the window of level wlvl, then the levels below it (lane quads, one line
// per query and level), then the leaf block.
template <typename K, typename V, typename W, int T, bool BOUND, bool KEEP>
__device__ __forceinline__ void bucket_item(const DevTree &t, const W *s_win, uint32_t w0, uint32_t wm,
                                            int wlvl, K base, const K *__restrict__ q, uint32_t qn,
                                            BktOut<V, BOUND> *__restrict__ out,
                                            uint8_t *__restrict__ found) {
    using LG = LeafGeom<K, V>;
    constexpr int U = sizeof(K) == 8 && !BOUND ? 2 : 4;  // queries per thread at a time
    const int lane = threadIdx.x & 31;
    const K tmax = (K)t.max_key;
    const unsigned char *leaves = static_cast<const unsigned char *>(t.leaves);
    for (uint32_t i0 = threadIdx.x & ~31u; i0 < qn; i0 += T * U) {
        K qv[U];
        W qw[U];
        uint32_t node[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const uint32_t i = i0 + u * T + lane;
            qv[u] = i < qn ? q[i] : (K)0;
            const K c = qv[u] < tmax ? qv[u] : tmax;
            if constexpr (sizeof(W) < sizeof(K)) {
                const K d = c > base ? c - base : (K)0;
                qw[u] = d < (K)0xFFFFFFFFu ? (W)d : (W)0xFFFFFFFFu;
            } else {
                qw[u] = c;
            }
        }
        win_bound<W, U>(s_win, wm, qw, node);
#pragma unroll
        for (int u = 0; u < U; u++) node[u] = w0 + (node[u] < wm ? node[u] : wm - 1u);
        if (wlvl + 1 < t.nlevels) {  // uniform: the window is not the bottom level
#pragma unroll 1
            for (int u = 0; u < U; u++) {
                K x = 0;
                uint32_t y = 0;
#pragma unroll
                for (int z = 0; z < U; z++)
                    if (z == u) {
                        x = qv[z];
                        y = node[z];
                    }
                y = walk_lanes<K, 4, 1>(t, wlvl + 1, x < tmax ? x : tmax, y, lane);
#pragma unroll
                for (int z = 0; z < U; z++) node[z] = z == u ? y : node[z];
            }
        }
        if constexpr (BOUND) {  // position of the first key at or above the query
            uint32_t w[U][8];
#pragma unroll
            for (int u = 0; u < U; u++) load_sector_as<KEEP>(leaves + (size_t)node[u] * LG::BS, w[u]);
#pragma unroll
            for (int u = 0; u < U; u++) {
                const K c = qv[u] < tmax ? qv[u] : tmax;
                const uint32_t i = i0 + u * T + lane;
                if (i < qn) out[i] = node[u] * (uint32_t)LG::S + count_below<K, LG::S>(w[u], c, false);
            }
        } else {
            leaf_answers<K, V, U, sizeof(K) == 8, KEEP>(leaves, node, qv, tmax, [&](int u, int l, V v, bool hit) {
                const uint32_t i = i0 + u * T + l;
                if (i < qn) {
                    out[i] = v;
                    if (found) found[i] = hit ? 1 : 0;
                }
            });
        }
    }
}

template <typename K, typename V, int T, bool BOUND, bool KEEP>
__global__ void __launch_bounds__(T, 1024 / T)
bucket_search_kernel(const __grid_constant__ DevTree t, const uint32_t *__restrict__ first,
                     const uint4 *__restrict__ items, const uint32_t *__restrict__ n_items,
                     uint32_t win_bytes, const K *__restrict__ q, BktOut<V, BOUND> *__restrict__ out,
                     uint8_t *__restrict__ found) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int F = kLineBytes / (int)sizeof(K);
    constexpr int LOGF = F == 32 ? 5 : 4;
    if (blockIdx.x >= *n_items) return;
    const uint4 it = items[blockIdx.x];
    const uint32_t blo = first[it.x], bhi = first[it.x + 1];
    const K *seps = static_cast<const K *>(t.seps);
    // the deepest level whose window fits; not more than 32 entries staged
    // per query (a line of the level per query)
    int wlvl = t.nlevels - 1, sh = 0;
    uint32_t w0, wm;
    const K *src;
    bool narrow;
    for (;;) {
        w0 = blo >> sh;
        wm = (bhi >> sh) - w0 + 1u;
        src = seps + t.lvl_off[wlvl] + w0;
        narrow = sizeof(K) == 4 || (uint64_t)src[wm - 1] - (uint64_t)src[0] < 0xFFFFFFFFull;
        if (wlvl == 0 || (win_words(wm) * (narrow ? 4 : 8) <= win_bytes && wm / 32 <= it.z)) break;
        wlvl--;
        sh += LOGF;
    }
    const K base = sizeof(K) == 8 && narrow ? src[0] : (K)0;
    if (narrow) {
        uint32_t *s_win = reinterpret_cast<uint32_t *>(smem_raw);
#pragma unroll 8
        for (uint32_t i = threadIdx.x; i < wm; i += T) s_win[win_slot(i)] = (uint32_t)(src[i] - base);
        __syncthreads();
        bucket_item<K, V, uint32_t, T, BOUND, KEEP>(t, s_win, w0, wm, wlvl, base, q + it.y, it.z, out + it.y,
                                       found ? found + it.y : nullptr);
    } else if constexpr (sizeof(K) == 8) {
        uint64_t *s_win = reinterpret_cast<uint64_t *>(smem_raw);
#pragma unroll 8
        for (uint32_t i = threadIdx.x; i < wm; i += T) s_win[win_slot(i)] = (uint64_t)src[i];
        __syncthreads();
        bucket_item<K, V, uint64_t, T, BOUND, KEEP>(t, s_win, w0, wm, wlvl, base, q + it.y, it.z, out + it.y,
                                       found ? found + it.y : nullptr);
    }
}

// Range bounds with the upper bound taken from the lower bound's path.
// A narrow range usually ends in the same bottom separator line as it
// starts: while the group walks lo down, it counts that line's separators
// <= hi as well (the line is already in its registers), which gives hi's
// leaf block whenever the line's last separator is above hi; both leaf
// blocks are then read together.  Only the queries whose range leaves that
// line take a second descent, compacted per warp into as few rounds as they
// need.  counts[i] = ub - lb (0 if lo > hi); lb_out[i] = lb.
template <typename K, typename V, int G, int R, bool PERM>
__global__ void __launch_bounds__(kThreads, 2)
bounds_line_kernel(const __grid_constant__ DevTree t, const K *__restrict__ lo,
                   const K *__restrict__ hi, const uint32_t *__restrict__ perm, uint64_t nq,
                   uint64_t *__restrict__ counts, uint64_t *__restrict__ lb_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    K *s_lvl = reinterpret_cast<K *>(smem_raw);
    stage_level<K>(s_lvl, t);
    __syncthreads();

    using LG = LeafGeom<K, V>;
    constexpr int F = kLineBytes / (int)sizeof(K);
    constexpr int KPL = F / G;
    constexpr int NB = KPL * (int)sizeof(K);
    constexpr int NG = 32 / G;
    constexpr int I = G / R;
    const int lane = threadIdx.x & 31;
    const int grp = lane / G;
    const int gl = lane % G;
    uint64_t *res = reinterpret_cast<uint64_t *>(smem_raw + scratch_offset(t)) + (threadIdx.x >> 5) * 64;
    const K tmax = (K)t.max_key;
    const unsigned char *leaves = static_cast<const unsigned char *>(t.leaves);
    const K *gseps = static_cast<const K *>(t.seps);
    const int bottom = t.nlevels - 1;
    // the staged level is the bottom one for small trees: no line to share
    const bool share = t.smem_level < bottom;
    const uint64_t ntiles = (nq + 31) / 32;
    const uint64_t per_cta = PERM ? (ntiles + gridDim.x - 1) / gridDim.x : 0;
    const uint64_t t_begin = PERM ? blockIdx.x * per_cta + (threadIdx.x >> 5)
                                  : (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t t_end = PERM ? min(ntiles, (blockIdx.x + 1) * per_cta) : ntiles;
    const uint64_t t_step = PERM ? (blockDim.x >> 5) : ((uint64_t)gridDim.x * blockDim.x) >> 5;

    for (uint64_t tile = t_begin; tile < t_end; tile += t_step) {
        const uint64_t base = tile * 32;
        const uint64_t my = base + lane;
        const bool v = my < nq;
        const K a = v ? lo[my] : (K)0;
        const K b = v ? hi[my] : (K)0;
        const K qa = a <= tmax ? a : tmax;
        const K qb = b < tmax ? b : tmax;
        const uint32_t na = smem_bound<K>(s_lvl, t.smem_entries, qa, false);
        // hi >= the largest key: the upper bound is n, no walk
        const bool hi_open = v && b < tmax;
        // ---- lower bounds, and upper bounds that end in the same bottom line
#pragma unroll
        for (int r = 0; r < R; r++) {
            K qe[2 * I];
            bool up[2 * I];
            uint32_t node[2 * I];
            bool hin[I];
#pragma unroll
            for (int s = 0; s < I; s++) {
                const int k = r * (NG * I) + s * NG + grp;
                qe[s] = __shfl_sync(0xffffffffu, qa, k);
                qe[I + s] = __shfl_sync(0xffffffffu, qb, k);
                node[s] = __shfl_sync(0xffffffffu, na, k);
                up[s] = false;
                up[I + s] = true;
                hin[s] = false;
            }
            for (int lvl = t.smem_level + 1; lvl < bottom; lvl++) {
                K qs[I];
                bool us[I];
                uint32_t ns[I];
#pragma unroll
                for (int s = 0; s < I; s++) {
                    qs[s] = qe[s];
                    us[s] = false;
                    ns[s] = node[s];
                }
                level_step<K, G, I>(gseps + t.lvl_off[lvl], qs, us, ns, grp, gl);
#pragma unroll
                for (int s = 0; s < I; s++) node[s] = ns[s];
            }
            if (share) {
                // bottom line: separators < lo and <= hi from the same registers
                uint32_t c[I][NB / 4];
#pragma unroll
                for (int s = 0; s < I; s++)
                    load_bytes<NB>(gseps + t.lvl_off[bottom] + (size_t)node[s] * F + gl * KPL, c[s]);
#pragma unroll
                for (int s = 0; s < I; s++) {
                    const int cl = group_count<G, G, KPL>(count_below<K, KPL>(c[s], qe[s], false), true, grp);
                    const int ch = group_count<G, G, KPL>(count_below<K, KPL>(c[s], qe[I + s], true), true, grp);
                    hin[s] = ch < F;  // the line's last separator is above hi
                    // (otherwise read lo's block again: ch = F may be past the last block)
                    node[I + s] = node[s] * F + (uint32_t)(hin[s] ? ch : cl);
                    node[s] = node[s] * F + (uint32_t)cl;
                }
            } else {
#pragma unroll
                for (int s = 0; s < I; s++) node[I + s] = node[s];
            }
            int pos[2 * I];
            leaf_bound<K, V, G, 2 * I>(leaves, node, qe, up, grp, gl, pos);
#pragma unroll
            for (int s = 0; s < I; s++) {
                const int k = r * (NG * I) + s * NG + grp;
                if (gl == 0) {
                    res[k] = (uint64_t)node[s] * LG::S + pos[s];
                    res[32 + k] = hin[s] ? (uint64_t)node[I + s] * LG::S + pos[I + s] : ~0ull;
                }
            }
        }
        __syncwarp();
        // ---- the remaining upper bounds: full descents, compacted
        const bool need = hi_open && res[32 + lane] == ~0ull;
        const unsigned needm = __ballot_sync(0xffffffffu, need);
        if (needm) {
            const uint32_t nb = need ? smem_bound<K>(s_lvl, t.smem_entries, qb, true) : 0u;
            const int nneed = __popc(needm);
            for (int r0 = 0; r0 < nneed; r0 += NG * I) {
                K qe[I];
                bool up[I];
                uint32_t node[I];
                int who[I];
#pragma unroll
                for (int s = 0; s < I; s++) {
                    const int j = r0 + s * NG + grp;  // j-th query that needs a descent
                    unsigned m = needm;               // its lane (the first one as filler)
                    for (int z = 0; z < (j < nneed ? j : 0); z++) m &= m - 1;
                    const int src = __ffs(m) - 1;
                    who[s] = j < nneed ? src : -1;
                    qe[s] = __shfl_sync(0xffffffffu, qb, src);
                    node[s] = __shfl_sync(0xffffffffu, nb, src);
                    up[s] = true;
                }
                walk_global<K, G, I>(t, qe, up, node, grp, gl);
                int pos[I];
                leaf_bound<K, V, G, I>(leaves, node, qe, up, grp, gl, pos);
#pragma unroll
                for (int s = 0; s < I; s++)
                    if (gl == 0 && who[s] >= 0) res[32 + who[s]] = (uint64_t)node[s] * LG::S + pos[s];
            }
        }
        __syncwarp();
        if (v) {
            const uint64_t lb = a <= tmax ? res[lane] : t.n;
            const uint64_t ub = b < tmax ? res[32 + lane] : t.n;
            const uint64_t dst = PERM ? (uint64_t)perm[my] : my;
            counts[dst] = (a <= b && ub > lb) ? ub - lb : 0;
            if (lb_out) lb_out[dst] = lb;
        }
        __syncwarp();
    }
}

// Empty tree: every point query misses, every range is empty.
template <typename V>
__global__ void fill_kernel(V *out, uint64_t n, V v) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = v;
}

std::mutex g_occ_mu;
std::map<std::pair<const void *, size_t>, int> g_occ;

// Resident CTAs per SM for a kernel at a given dynamic shared memory size
// (all devices this library runs on are B200s of one kind).
int occupancy(const void *fn, size_t smem) {
    std::lock_guard<std::mutex> lk(g_occ_mu);
    auto key = std::make_pair(fn, smem);
    auto it = g_occ.find(key);
    if (it != g_occ.end()) return it->second;
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, fn, kThreads, smem) != cudaSuccess ||
        blocks < 1)
        blocks = 1;
    g_occ[key] = blocks;
    return blocks;
}

unsigned persistent_grid(const void *fn, size_t smem, uint64_t work_items, uint64_t items_per_cta) {
    uint64_t want = (work_items + items_per_cta - 1) / items_per_cta;
    uint64_t cap = (uint64_t)sm_count() * occupancy(fn, smem);
    if (want > cap) want = cap;
    return (unsigned)(want < 1 ? 1 : want);
}

// Raises a kernel's dynamic shared-memory limit when needed (function
// attributes are per device; the largest size set so far is remembered).
template <typename Fn>
bt_status set_smem(Fn fn, size_t smem) {
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, size_t> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_pair(dev, (const void *)fn);
    auto it = done.find(key);
    if (it != done.end() && it->second >= smem) return BT_OK;
    if (smem > 48 * 1024)
        BT_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    done[key] = smem;
    return BT_OK;
}

template <typename K, typename V, int G, int R, bool PERM, bool PAIR>
bt_status point_launch_t(const bt_tree *t, const void *d_q, const uint32_t *d_perm, uint64_t nq,
                         void *d_out, uint8_t *d_found, cudaStream_t s) {
    auto fn = point_kernel<K, V, G, R, PERM, PAIR>;
    const size_t smem = win_words(t->dev.smem_entries) * sizeof(K);
    bt_status st = set_smem(fn, smem);
    if (st != BT_OK) return st;
    const unsigned grid = persistent_grid((const void *)fn, smem, nq, kThreads);
    count_launch();
    fn<<<grid, kThreads, smem, s>>>(t->dev, (const K *)d_q, d_perm, nq, (V *)d_out, d_found);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

// Leaf arrays above this are read by lane pairs also with 4-byte keys: a block
// that comes from DRAM is then one request for both sectors (2^26 keys, 2^21
// queries: 80 us a call; a thread per query 110; four lanes per query 84), where one
// from L2 is faster by a thread (2^20 keys, 2^20 queries: 25.8 us; pairs 28.0;
// four lanes 36).  The lines cross between 2^23 and 2^24 keys (64 / 128 MiB).
constexpr size_t kPairLeafBytes = 64ull << 20;

template <typename K, typename V, int G, int R, bool PERM>
bt_status point_launch(const bt_tree *t, const void *d_q, const uint32_t *d_perm, uint64_t nq,
                       void *d_out, uint8_t *d_found, cudaStream_t s) {
    using LG = LeafGeom<K, V>;
    if constexpr (sizeof(K) == 8)
        return point_launch_t<K, V, G, R, PERM, true>(t, d_q, d_perm, nq, d_out, d_found, s);
    if constexpr (LG::BS == 2 * kSectorBytes)
        if (t->n_sectors * LG::BS > kPairLeafBytes)
            return point_launch_t<K, V, G, R, PERM, LG::BS == 2 * kSectorBytes>(t, d_q, d_perm, nq, d_out, d_found, s);
    return point_launch_t<K, V, G, R, PERM, false>(t, d_q, d_perm, nq, d_out, d_found, s);
}

// One shape per key width, whatever the tree's is set to: that is chosen on
// point_kernel, whose best differs (2^24 grouped queries, us: u32 2^26 keys (4,1)
// 560 (4,2) 591 (8,2) 753 (2,1) 847 (8,1) 1080; u64 2^28 keys (4,2) 1317 (4,1)
// 1335 (2,1) 1389 (8,2) 1501 (8,1) 1834; the same order at 2^22 queries).
template <typename K, typename V>
bt_status window_launch(const bt_tree *t, const void *d_q, const uint32_t *d_perm, uint64_t nq,
                        void *d_out, uint8_t *d_found, cudaStream_t s) {
    auto fn = point_window_kernel<K, V, 4, sizeof(K) == 4 ? 1 : 2>;
    bt_status st = set_smem(fn, kWinBytes);
    if (st != BT_OK) return st;
    const uint64_t ntiles = (nq + 31) / 32;
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ntiles, sm_count()));
    const int shift = std::max(0, bitlen64(t->max_key) - kPointGroupBits);  // as the grouping pass
    count_launch();
    fn<<<grid, kWinThreads, kWinBytes, s>>>(t->dev, (const K *)d_q, d_perm, nq, (V *)d_out, d_found,
                                            shift);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

template <typename K, typename V, int T, bool BOUND, bool KEEP = false>
bt_status bucket_launch(const bt_tree *t, const BucketPlan &bp, uint64_t max_items, size_t smem,
                        const void *d_q, void *d_out, uint8_t *d_found, cudaStream_t s) {
    auto fn = bucket_search_kernel<K, V, T, BOUND, KEEP>;
    bt_status st = set_smem(fn, smem);
    if (st != BT_OK) return st;
    count_launch();
    fn<<<(unsigned)max_items, T, smem, s>>>(t->dev, bp.first, bp.items, bp.n_items, (uint32_t)smem,
                                            (const K *)d_q, (BktOut<V, BOUND> *)d_out, d_found);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

template <typename K, typename V, bool BOUND>
bt_status bucket_cfg(const bt_tree *t, const BucketPlan &bp, uint64_t max_items,
                     const void *d_q, void *d_out, uint8_t *d_found, cudaStream_t s) {
    // the fullest bucket's window of the deepest level that fits, in 32-bit
    // entries (the kernel goes a level up where its own does not)
    constexpr int LOGF = sizeof(K) == 4 ? 5 : 4;
    size_t m = t->bucket_blocks;
    while (win_words(m) * sizeof(uint32_t) > kBktWinBytes) m = (m >> LOGF) + 2;
    const size_t smem = std::max<size_t>(win_words(m) * sizeof(uint32_t), kBktWinMin);
    if (t->bucket_blocks <= kKeepBlocks)
        return bucket_launch<K, V, 512, BOUND, true>(t, bp, max_items, smem, d_q, d_out, d_found, s);
    // two CTAs per SM where two windows fit
    if (smem <= kBktWinBytes / 2) return bucket_launch<K, V, 512, BOUND>(t, bp, max_items, smem, d_q, d_out, d_found, s);
    return bucket_launch<K, V, 1024, BOUND>(t, bp, max_items, smem, d_q, d_out, d_found, s);
}

template <typename K, typename V, bool PERM>
bt_status point_cfg(const bt_tree *t, const void *d_q, const uint32_t *d_perm, uint64_t nq,
                    void *d_out, uint8_t *d_found, cudaStream_t s) {
    if (PERM && nq >= kWinMinQueries) return window_launch<K, V>(t, d_q, d_perm, nq, d_out, d_found, s);
    switch (shape_of(t, BT_OP_POINT, nq)) {
        case 0: return point_launch<K, V, 8, 1, PERM>(t, d_q, d_perm, nq, d_out, d_found, s);
        case 1: return point_launch<K, V, 8, 2, PERM>(t, d_q, d_perm, nq, d_out, d_found, s);
        case 2: return point_launch<K, V, 4, 1, PERM>(t, d_q, d_perm, nq, d_out, d_found, s);
        case 3: return point_launch<K, V, 4, 2, PERM>(t, d_q, d_perm, nq, d_out, d_found, s);
        default: return point_launch<K, V, 2, 1, PERM>(t, d_q, d_perm, nq, d_out, d_found, s);
    }
}

template <typename K, typename V, int G, int R, bool PERM>
bt_status bounds_launch(const bt_tree *t, const void *d_lo, const void *d_hi,
                        const uint32_t *d_perm, uint64_t nq, uint64_t *d_counts, uint64_t *d_lb,
                        cudaStream_t s) {
    auto fn = bounds_line_kernel<K, V, G, R, PERM>;
    const size_t smem = scratch_offset(t->dev) + (size_t)kWarps * 64 * sizeof(uint64_t);
    bt_status st = set_smem(fn, smem);
    if (st != BT_OK) return st;
    const unsigned grid = persistent_grid((const void *)fn, smem, nq, kThreads);
    count_launch();
    fn<<<grid, kThreads, smem, s>>>(t->dev, (const K *)d_lo, (const K *)d_hi, d_perm, nq, d_counts,
                                    d_lb);
    BT_CUDA(cudaGetLastError());
    return BT_OK;
}

template <typename K, typename V, bool PERM>
bt_status bounds_cfg(const bt_tree *t, const void *d_lo, const void *d_hi, const uint32_t *d_perm,
                     uint64_t nq, uint64_t *d_counts, uint64_t *d_lb, cudaStream_t s) {
    switch (shape_of(t, BT_OP_RANGE, nq)) {
        case 0: return bounds_launch<K, V, 8, 1, PERM>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s);
        case 1: return bounds_launch<K, V, 8, 2, PERM>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s);
        case 2: return bounds_launch<K, V, 4, 1, PERM>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s);
        case 3: return bounds_launch<K, V, 4, 2, PERM>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s);
        default: return bounds_launch<K, V, 2, 1, PERM>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s);
    }
}

template <bool PERM>
bt_status point_types(const bt_tree *t, const void *d_q, const uint32_t *d_perm, uint64_t nq,
                      void *d_out, uint8_t *d_found, cudaStream_t s) {
    if (t->key_bytes == 4)
        return t->val_bytes == 4 ? point_cfg<uint32_t, uint32_t, PERM>(t, d_q, d_perm, nq, d_out, d_found, s)
                                 : point_cfg<uint32_t, uint64_t, PERM>(t, d_q, d_perm, nq, d_out, d_found, s);
    return t->val_bytes == 4 ? point_cfg<uint64_t, uint32_t, PERM>(t, d_q, d_perm, nq, d_out, d_found, s)
                             : point_cfg<uint64_t, uint64_t, PERM>(t, d_q, d_perm, nq, d_out, d_found, s);
}

template <bool PERM>
bt_status bounds_types(const bt_tree *t, const void *d_lo, const void *d_hi, const uint32_t *d_perm,
                       uint64_t nq, uint64_t *d_counts, uint64_t *d_lb, cudaStream_t s) {
    if (t->key_bytes == 4)
        return t->val_bytes == 4
                   ? bounds_cfg<uint32_t, uint32_t, PERM>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s)
                   : bounds_cfg<uint32_t, uint64_t, PERM>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s);
    return t->val_bytes == 4
               ? bounds_cfg<uint64_t, uint32_t, PERM>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s)
               : bounds_cfg<uint64_t, uint64_t, PERM>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s);
}

}  // namespace

bt_status launch_point_search(const bt_tree *t, const void *d_q, const uint32_t *d_perm,
                              uint64_t nq, void *d_out, cudaStream_t s, uint8_t *d_found) {
    if (nq == 0) return BT_OK;
    if (t->n == 0) {
        unsigned g = (unsigned)std::min<uint64_t>((nq + 255) / 256, 4096);
        count_launch();
        if (t->val_bytes == 4)
            fill_kernel<uint32_t><<<g, 256, 0, s>>>((uint32_t *)d_out, nq, 0xFFFFFFFFu);
        else
            fill_kernel<uint64_t><<<g, 256, 0, s>>>((uint64_t *)d_out, nq, ~0ull);
        BT_CUDA(cudaGetLastError());
        if (d_found) BT_CUDA(cudaMemsetAsync(d_found, 0, nq, s));
        return BT_OK;
    }
    return d_perm ? point_types<true>(t, d_q, d_perm, nq, d_out, d_found, s)
                  : point_types<false>(t, d_q, d_perm, nq, d_out, d_found, s);
}

// Trees whose keys crowd into few of the equal stretches (a bucket of over four
// times the average) keep the direct search: the windows of the full ones lie
// levels above the leaves.  Half the keys in 1 / 2R of the range, so that the
// fullest bucket is R times the average one, direct / by buckets (us):
//   u64, 2^26, 2^22 queries   R 1.5 250 / 240   2.5 250 / 243   3.5 248 / 287   6.5 250 / 282
//              2^24 queries         898 / 707       898 / 689       898 / 730       899 / 857
//              2^22 ranges          392 / 405       390 / 399       391 / 442       390 / 487
//   u64, 2^24, 2^22 queries         223 / 218       222 / 213       224 / 217  16.6 225 / 256
// (learned batches gain up to R 16, where their index fits: 1079 / 768.)  So does
// a stream under capture, whose graph then holds no allocation.  And the passes
// must pay for the separators staged: every query for eight leaf blocks (2^23
// queries at 2^28 u64 keys: 674 us directly, 515 by buckets).
static bool buckets_suit(const bt_tree *t, uint64_t nq, uint64_t blocks_per_query, cudaStream_t s) {
    if (t->n == 0 || nq >= (1ull << 32) || nq < t->n_sectors / blocks_per_query) return false;
    const uint64_t buckets = bucket_map(t->min_key, t->max_key).last + 1;
    if (t->bucket_blocks == 0 || t->bucket_blocks > 4 * (t->n_sectors / buckets) + 64) return false;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone) return true;
    cudaGetLastError();
    return false;
}

// Point searches, direct / by buckets (us, whole calls on uniform queries):
//                 2^21 queries   2^22       2^23       2^24
//   u32, 2^16                    78 / 108   128 / 166  238 / 274
//   u32, 2^18                    98 / 113   174 / 172  326 / 289
//   u32, 2^22                   109 / 130   189 / 190  347 / 324
//   u32, 2^23                   134 / 133   239 / 199  450 / 333
//   u32, 2^26      98 / 108     166 / 163              607 / 392
//   u64, 2^14                    93 / 141   164 / 240  308 / 400
//   u64, 2^18                   132 / 148   240 / 246  458 / 422
//   u64, 2^20      91 / 97      164 / 155   302 / 253  583 / 441
//   u64, 2^26     137 / 149     249 / 213             1056 / 544
// (u64, 2^18: 4 us a million queries one way or the other, but 352 / 132 where
// they fall on 64 keys.)  The SMs of a direct u64 search of a tree of a few leaf
// blocks wait for the same L2 lines:
//   blocks           5          13         25        50        100       200
//   2^20 queries    37 / 66    96 / 66    70 / 60   51 / 62   33 / 70   25 / 62
//   2^21            68 / 90   182 / 86   133 / 80   92 / 84   59 / 88   43 / 82
//   2^22           125 / 133  354 / 125  256 / 119 174 / 121 108 / 131  74 / 123
// (u32, 13 to 25 blocks: 45 / 88 at 2^22.)  75 blocks, 2^24 queries: uniform 452 / 350,
// Zipf 729 / 346; 250: 284 / 344, 279 / 350.  Larger ones up to 1 MiB lose only where a
// batch falls on neighbouring keys (64 of them, 2^22 queries: 328 / 130).
bool point_order_pays(const bt_tree *t, uint64_t nq) {
    if (t->key_bytes == 8 && t->n_sectors > 8 && t->n_sectors <= 128)
        return nq >= (t->n_sectors <= 64 ? 1ull << 21 : 1ull << 22);
    const uint64_t bytes = t->n_sectors * (uint64_t)leaf_stride(t->key_bytes, t->val_bytes);
    if (bytes <= 1ull << 20) return false;  // in L1 without any order
    return nq >= (t->key_bytes == 4 && bytes <= kPairLeafBytes ? 1ull << 23 : 1ull << 22);
}

bool bucket_search_pays(const bt_tree *t, uint64_t nq, cudaStream_t s) {
    return point_order_pays(t, nq) && buckets_suit(t, nq, 8, s);
}

// Learned searches: how many queries pay for the order depends on how far the
// direct kernel's rank windows reach (learned_least).
bool learned_buckets_pay(const bt_tree *t, uint64_t nq, cudaStream_t s) {
    return nq >= learned_least(t) && buckets_suit(t, nq, ~0ull, s) && learned_index_fits(t);
}

// Range bounds, direct / by buckets (us; the buckets take both bounds of a
// range as queries of their own, so its width does not matter), uniform ranges
// and (sorted ones):
//                    2^20 ranges          1.5 * 2^20           2^21                 2^22
//   u32, 2^20 keys   56 / 95 (48 / 87)    72 / 116 (62 / 98)   91 / 126 (76 / 113)  157 / 198 (126 / 178)
//   u32, 2^24        77 / 110 (63 / 106) 105 / 130 (83 / 118) 132 / 147 (103 / 135) 236 / 217 (176 / 199)
//   u32, 2^26        92 / 124 (80 / 119) 126 / 147 (108 / 140) 154 / 167 (130 / 158) 276 / 244 (229 / 230)
//   u64, 2^20       100 / 107 (79 / 100) 144 / 125 (106 / 113) 179 / 158 (138 / 140) 332 / 245 (227 / 232)
//   u64, 2^26       134 / 154 (114 / 153) 191 / 181 (158 / 176) 238 / 221 (192 / 214) 442 / 336 (343 / 327)
// On few keys the buckets gain more (2^22 ranges from 256 of 2^20 u32 keys: 415 / 182),
// and on few leaf blocks, whose lines all SMs then wait for:
//   blocks                 7         13        25        50       100       200
//   2^20 ranges, u32    80 / 58  188 / 58  170 / 58  117 / 62   74 / 62   45 / 64
//   2^20 ranges, u64   166 / 68  281 / 66  207 / 66  141 / 66   86 / 70   66 / 68
//   2^19, u32           45 / 52   98 / 49   90 / 49   64 / 49   41 / 53
bool range_order_pays(const bt_tree *t, uint64_t nr) {
    if (t->n_sectors <= 128) return nr >= 1ull << 20;
    return nr >= (t->key_bytes == 4 ? 1ull << 22 : 3ull << 19);
}

bool bucket_bounds_pay(const bt_tree *t, uint64_t nr, cudaStream_t s) {
    return range_order_pays(t, nr) && nr < (1ull << 31) && t->n < (1ull << 32) && buckets_suit(t, 2 * nr, 8, s);
}

namespace {
template <bool BOUND>
bt_status bucket_types(const bt_tree *t, const BucketWs &w, cudaStream_t s) {
    if (t->key_bytes == 4)
        return t->val_bytes == 4
                   ? bucket_cfg<uint32_t, uint32_t, BOUND>(t, w.bp, w.max_items, w.q, w.res, w.found, s)
                   : bucket_cfg<uint32_t, uint64_t, BOUND>(t, w.bp, w.max_items, w.q, w.res, w.found, s);
    return t->val_bytes == 4
               ? bucket_cfg<uint64_t, uint32_t, BOUND>(t, w.bp, w.max_items, w.q, w.res, w.found, s)
               : bucket_cfg<uint64_t, uint64_t, BOUND>(t, w.bp, w.max_items, w.q, w.res, w.found, s);
}
}  // namespace

bt_status launch_bucket_search(const bt_tree *t, const void *d_q, uint64_t nq, void *d_out,
                               cudaStream_t s, uint8_t *d_found) {
    const BucketMap map = bucket_map(t->min_key, t->max_key);
    const uint64_t per = bucket_batch(t, nq);
    BucketWs w(s);
    bt_status st = w.alloc(per, map.last + 1, t->key_bytes, t->val_bytes, d_found != nullptr);
    for (uint64_t i = 0; i < nq && st == BT_OK; i += per) {
        const uint64_t m = std::min(per, nq - i);
        st = launch_buckets(t, map, (const char *)d_q + i * t->key_bytes, nullptr, m, w.q, w.pos, w.bp, s);
        if (st == BT_OK) st = bucket_types<false>(t, w, s);
        if (st == BT_OK)
            st = launch_bucket_gather(t->val_bytes, w.res, w.found, w.pos, m, (char *)d_out + i * t->val_bytes,
                                      d_found ? d_found + i : nullptr, s);
    }
    return st;
}

bt_status launch_bucket_bounds(const bt_tree *t, const void *d_lo, const void *d_hi, uint64_t nr,
                               uint64_t *d_counts, uint64_t *d_lb, cudaStream_t s) {
    const BucketMap map = bucket_map(t->min_key, t->max_key);
    const uint64_t per = (bucket_batch(t, 2 * nr) + 1) / 2;
    BucketWs w(s);
    bt_status st = w.alloc(2 * per, map.last + 1, t->key_bytes, sizeof(uint32_t), false);
    for (uint64_t i = 0; i < nr && st == BT_OK; i += per) {
        const uint64_t m = std::min(per, nr - i);
        const char *lo = (const char *)d_lo + i * t->key_bytes, *hi = (const char *)d_hi + i * t->key_bytes;
        st = launch_buckets(t, map, lo, hi, m, w.q, w.pos, w.bp, s);
        if (st == BT_OK) st = bucket_types<true>(t, w, s);
        if (st == BT_OK)
            st = launch_range_gather(t, reinterpret_cast<const uint32_t *>(w.res), w.pos, lo, hi, m,
                                     d_counts + i, d_lb ? d_lb + i : nullptr, s);
    }
    return st;
}

bt_status launch_bounds(const bt_tree *t, const void *d_lo, const void *d_hi,
                        const uint32_t *d_perm, uint64_t nq, uint64_t *d_counts, uint64_t *d_lb,
                        cudaStream_t s) {
    if (nq == 0) return BT_OK;
    if (t->n == 0) {
        unsigned g = (unsigned)std::min<uint64_t>((nq + 255) / 256, 4096);
        count_launch();
        fill_kernel<uint64_t><<<g, 256, 0, s>>>(d_counts, nq, 0ull);
        if (d_lb) {
            count_launch();
            fill_kernel<uint64_t><<<g, 256, 0, s>>>(d_lb, nq, 0ull);
        }
        BT_CUDA(cudaGetLastError());
        return BT_OK;
    }
    return d_perm ? bounds_types<true>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s)
                  : bounds_types<false>(t, d_lo, d_hi, d_perm, nq, d_counts, d_lb, s);
}

}  // namespace bt
