// Internal definitions shared by the engine's translation units.
//
// Tree layout in HBM (one allocation per array, 256-byte aligned):
//
//   leaves  the sorted keys and their values in leaf blocks.  Block b holds
//           keys b*S .. b*S+S-1 (S = 32 / sizeof(key): one 32-byte DRAM
//           sector) followed by the same positions' values, the block padded
//           to a power of two (64 bytes, or 128 for 4-byte keys with 8-byte
//           values).  A point-search hit needs one block: its key sector and
//           value sector come in the same 64-byte DRAM access.  Unused key
//           slots of the last block hold the all-ones key.
//   seps    separator levels, stored root first.  Level t holds nodes of
//           F = 128 / sizeof(key) separators (one 128-byte line).  A
//           separator is the maximum key of the node (or leaf block) below
//           it, as in the reference's internal pages (BPTree.cu:54-55).
//
// Child j of node i at level t is node i*F + j of level t+1; the children of
// the bottom level are leaf blocks.  No pointers are stored.  A search for
// q <= max_key takes, at every level, the first separator >= q (lower bound)
// or > q (upper bound); padding separators are all-ones and never win.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <string>

#include "../../include/btree_b200.h"

#define BT_VERSION_NUMBER 10000

namespace bt {

constexpr int kLineBytes = 128;   // internal node size
constexpr int kSectorBytes = 32;  // leaf sector size
constexpr int kMaxLevels = 24;

// Shared-memory budget for the separator level a search CTA stages (the
// deepest level that fits is staged and binary-searched per query).
constexpr size_t kSmemTopBudget = 96 * 1024;

// Leaf block geometry for key type K and value type V.
template <typename K, typename V>
struct LeafGeom {
    static constexpr int S = kSectorBytes / (int)sizeof(K);  // keys per block
    static constexpr int VB = S * (int)sizeof(V);             // value bytes per block
    static constexpr int BS = (kSectorBytes + VB) <= 64 ? 64 : 128;  // block stride
};

inline int leaf_stride(int key_bytes, int val_bytes) {
    const int vb = (kSectorBytes / key_bytes) * val_bytes;
    return (kSectorBytes + vb) <= 64 ? 64 : 128;
}

struct DevTree {
    const void *leaves;
    const void *seps;
    uint64_t n;
    uint64_t max_key;
    uint64_t n_sectors;
    uint64_t lvl_off[kMaxLevels];  // element offset of level t in seps (t = 0 is the root)
    int nlevels;
    int smem_level;                // level staged in shared memory (resolves levels 0..smem_level)
    uint32_t smem_entries;         // its real separators
    uint32_t smem_bytes;           // bytes staged (a multiple of 16)
};

// ---- learned index (see bt_learned.cu) ----------------------------------

constexpr int kSegPerLine = 4;      // segments per segment line
constexpr int kCodesPerLine = 59;   // thresholds per code line
constexpr int kUnitBytes = 128;     // a leaf unit: the 128-byte aligned piece of the leaf array

// One segment (leaf model): it covers the keys [key, next segment's key),
// ranks r_lo .. r_lo + cnt - 1; rank ~ r_lo + clamp(icpt + slope * (q -
// key), 0, cnt) within eps of the truth for every key of the segment.
struct SegRec {
    uint64_t key;
    uint32_t r_lo, cnt;
    float slope, icpt;
    uint32_t eps, pad;
};

// Four consecutive segments in one 128-byte line, 32 bytes each, so that
// each lane of a pair reading a 64-byte half holds two whole segments.
// Unused slots of the last line: key all-ones, r_lo = n, cnt = 0.
struct SegLine {
    SegRec s[kSegPerLine];
};

// Thresholds between consecutive leaf units, 59 per 128-byte line.
// Threshold j separates unit j from unit j + 1: T_j = base + (code << shift)
// is the smallest such value above the largest key of unit j, so q >= T_j
// iff q >= base and ((q - base) >> shift) >= code.  Codes are 15-bit values
// (at most kCodeMax; kCodePad marks a slot past the last threshold), so that
// two of them in a 32-bit word compare against the key in one subtraction.
constexpr uint32_t kCodeMax = 0x7FFEu;
constexpr uint32_t kCodePad = 0x7FFFu;

struct CodeLine {
    uint64_t base;
    uint16_t shift;
    uint16_t code[kCodesPerLine];
};

constexpr int kMaxHidden = 32;

// Device view of a trained learned index.
struct LearnedDev {
    const float *mlp;        // root parameters (3*hidden+1)
    const SegLine *seg;      // segment lines
    const CodeLine *codes;   // code lines
    const void *stage;       // first key of every segment line (key type), nls entries
    unsigned long long *stats;  // [extra leaf-unit reads, full-descent fallbacks] of the last search
    uint64_t kmin;           // root input: x = (key - kmin) * xscale
    float xscale;
    int hidden;
    uint32_t nseg;           // segments
    uint32_t nls;            // segment lines
    uint32_t root_err;       // |root's line prediction - line| <= root_err at every staged key
    uint32_t kpu;            // keys per leaf unit
    uint64_t units;          // leaf units
    const uint32_t *seg_first;  // first segment that a query of bucket b can route to, b = 0 .. last + 1
    uint32_t stage_bytes;    // shared-memory bytes of the staged keys (whole bank rows)
};

struct LearnedState;

}  // namespace bt

struct bt_tree {
    int device;
    int key_bytes;
    int val_bytes;
    uint64_t n;
    uint64_t n_sectors;
    void *d_leaves;
    void *d_seps;
    uint64_t seps_elems;
    uint64_t lvl_nodes[bt::kMaxLevels];
    uint64_t lvl_entries[bt::kMaxLevels];
    uint64_t min_key, max_key;
    int values_sorted;
    uint32_t bucket_blocks;  // leaf blocks of the fullest bucket (0: not measured)
    int search_cfg[2];  // per bt_search_op: index into the (lanes, rounds) table, -1: own_search_cfg
    bt::DevTree dev;
    bt::LearnedState *learned;  // trained learned index, or null
};

namespace bt {

// Thread-local error detail, set by fail().
void set_error(const std::string &msg);
bt_status fail(bt_status s, const std::string &msg);
bt_status cuda_fail(cudaError_t e, const char *what);

#define BT_CUDA(call)                                            \
    do {                                                         \
        cudaError_t e__ = (call);                                \
        if (e__ != cudaSuccess) return ::bt::cuda_fail(e__, #call); \
    } while (0)

// Stream-ordered allocation from the engine's own memory pool on the
// current device (cached between calls, never returned to other users).
bt_status ws_alloc(void **p, size_t bytes, cudaStream_t s);
void ws_free(void *p, cudaStream_t s);

// A workspace allocation returned to the pool (stream-ordered) when the
// guard leaves scope, on every path out of the function.
struct WsGuard {
    void *p = nullptr;
    cudaStream_t s;
    explicit WsGuard(cudaStream_t st) : s(st) {}
    WsGuard(const WsGuard &) = delete;
    WsGuard &operator=(const WsGuard &) = delete;
    ~WsGuard() {
        if (p) ws_free(p, s);
    }
    bt_status alloc(size_t bytes) { return ws_alloc(&p, bytes, s); }
    template <typename T>
    T *as() const { return static_cast<T *>(p); }
};

// Counts one kernel launch (bt_kernel_launches).
void count_launch();
// Number of SMs of the current device (cached).
int sm_count();
// Checks the current device is sm_100 class.
bt_status require_device(int device);

template <typename K>
__host__ __device__ constexpr K key_max() {
    return (K)~(K)0;
}

__host__ __device__ inline int bitlen64(uint64_t v) {
    int b = 0;
    while (v) {
        v >>= 1;
        b++;
    }
    return b;
}

// The point search behind bt_point_search (arguments checked, the tree's device
// current, the learned counters reset).  `scratch`: whether it may order a large
// batch, by bucket or in groups.
bt_status point_device(const bt_tree *t, int mode, const void *d_q, uint64_t nq, void *d_out,
                       cudaStream_t s, uint8_t *d_found, bool scratch);
// Host launchers implemented in the .cu files.
bt_status launch_point_search(const bt_tree *t, const void *d_q, const uint32_t *d_perm,
                              uint64_t nq, void *d_out, cudaStream_t s,
                              uint8_t *d_found = nullptr);
bt_status launch_bounds(const bt_tree *t, const void *d_lo, const void *d_hi,
                        const uint32_t *d_perm, uint64_t nq, uint64_t *d_counts,
                        uint64_t *d_lb, cudaStream_t s);
bt_status launch_partition(const bt_tree *t, int kind, const void *d_a, const void *d_b,
                           uint64_t nq, void *d_out_a, void *d_out_b, uint32_t *d_perm,
                           cudaStream_t s);
// d_total: two words, the sum and the largest input.
bt_status launch_scan_u64(const uint64_t *d_in, uint64_t *d_out, uint64_t n, uint64_t *d_total,
                          cudaStream_t s);
// Point-query partition into caller memory: ws must hold
// partition_point_ws_bytes(nq) bytes; nothing is allocated.
size_t partition_point_ws_bytes(uint64_t nq);
bt_status launch_partition_point_prealloc(const bt_tree *t, const void *d_q, uint64_t nq,
                                          void *out_q, uint32_t *out_perm, void *ws,
                                          cudaStream_t s);
// IDs of every range, sorted ascending; max_count = the largest count.
bt_status launch_range_fill(const bt_tree *t, const uint64_t *d_lb, const uint64_t *d_counts,
                            const uint64_t *d_offsets, uint64_t nq, uint64_t max_count, void *d_ids,
                            cudaStream_t s);
// Stable sort of n (key, value) pairs by key on the device: LSD radix sort
// with 8-bit digits (key_bytes passes of the partition kernels, the values
// carried with their keys).  Equal keys keep their input order.  Scratch: one
// copy of the pairs and a table.  n < 2^32; outputs must not alias inputs.
bt_status launch_sort_pairs(int key_bytes, int value_bytes, const void *d_keys, const void *d_vals,
                            uint64_t n, void *out_keys, void *out_vals, cudaStream_t s);
// Stable order of n 16-bit keys (the low halves of d_keys): d_perm[g] = the
// index of the item in position g (two 8-bit passes of the partition).
bt_status launch_order_u16(const uint32_t *d_keys, uint64_t n, uint32_t *d_perm, cudaStream_t s);
// Sorts the segments ids[offsets[i] .. + counts[i]) longer than 256 values
// (shorter ones are sorted as they are written); max_count = the largest.
bt_status launch_segment_sort(const bt_tree *t, const uint64_t *d_counts, const uint64_t *d_offsets,
                              uint64_t nseg, uint64_t max_count, void *d_ids, cudaStream_t s);

// (lanes per query, rounds) -> index of the search configuration table in
// bt_search.cu, or -1.
int search_cfg_index(int lanes, int rounds);
// The shape in which nq queries or ranges are searched on a tree whose own is
// not set.
int own_search_cfg(int key_bytes, int op, uint64_t nq);
int search_cfg_lanes(int cfg);
int search_cfg_rounds(int cfg);

// Where a search writes its `total` > 0 IDs: the caller's buffer if it is
// large enough, or what the caller's function returns.  Null: *st says why.
inline void *ids_buffer(void *ids, uint64_t capacity, uint64_t total, bt_status *st) {
    if (total > capacity) *st = fail(BT_ERR_CAPACITY, "ids_capacity is below the total hit count");
    else if (!ids) *st = fail(BT_ERR_INVALID_ARGUMENT, "ids is NULL");
    else return ids;
    return nullptr;
}
inline void *ids_from(bt_ids_alloc alloc, void *ctx, uint64_t total, bt_status *st) {
    void *ids = alloc(ctx, total);
    if (!ids) *st = fail(BT_ERR_OUT_OF_MEMORY, "the ID allocation function returned NULL");
    return ids;
}

void free_learned(bt::LearnedState *s);
// Learned point search of d_q into d_out on s (the tree has a learned index;
// the counters of bt_learned_last_stats accumulate).
bt_status launch_learned_search(const bt_tree *t, const void *d_q, uint64_t nq, void *d_out,
                                uint8_t *d_found, cudaStream_t s);
// Whether the bucket search's shared memory holds every bucket's part of the
// tree's learned index.
bool learned_index_fits(const bt_tree *t);
// The least batch that pays for the bucket order on the tree's learned index.
uint64_t learned_least(const bt_tree *t);
// The same for a batch that learned_buckets_pay for, ordered by bucket
// (BT_ERR_OUT_OF_MEMORY when the workspace cannot be had).
bt_status launch_learned_buckets(const bt_tree *t, const void *d_q, uint64_t nq, void *d_out,
                                 uint8_t *d_found, cudaStream_t s);
// Zeroes those counters (stream-ordered).
bt_status reset_learned_stats(const bt_tree *t, cudaStream_t s);

// Buckets of a point batch: equal stretches of the tree's key range
// [min, max], numbered by the key's offset from the smallest key shifted
// right; keys outside the range go to the end buckets.
constexpr int kMaxBuckets = 2048;
struct BucketMap {
    uint64_t min;
    int shift;
    uint32_t last;  // the highest bucket
    template <typename K>
    __device__ __forceinline__ uint32_t of(K k) const {
        const K d = k > (K)min ? k - (K)min : (K)0;
        const K b = d >> shift;
        return b < (K)last ? (uint32_t)b : last;
    }
    __device__ __forceinline__ uint64_t first_key(uint32_t b) const {
        return b == 0 ? 0ull : min + ((uint64_t)b << shift);
    }
};
// Most queries of one work item of the bucket search; fewer in a batch that falls
// on few buckets, so that its items still fill the GPU's 296 CTAs (2^20 u64 keys,
// 2^18 learned queries for 64 of them: 111 -> 67 us).
constexpr uint32_t kBucketSlice = 16384;
constexpr uint32_t kBucketMinSlice = 1024;
inline uint32_t bucket_slice(uint64_t nq) {
    return (uint32_t)std::min<uint64_t>(kBucketSlice, std::max<uint64_t>(kBucketMinSlice, nq / 512));
}
// What the passes of the bucket order leave for the search.
struct BucketPlan {
    uint32_t *scratch;  // 2 * kMaxBuckets words
    uint32_t *first;    // leaf block where bucket b's keys start, b = 0 .. last; last + 1: of the largest key
    uint4 *items;       // work items: bucket, first slot, slots
    uint32_t *n_items;  // at most kMaxBuckets + nq / bucket_slice(nq)
};
// d_q ordered by bucket into out_q (query i in slot pos[i]).  With d_hi, the
// 2 nq bounds of the ranges [d_q[i], d_hi[i]]: d_q[i], then d_hi[i] + 1.
bt_status launch_buckets(const bt_tree *t, const BucketMap &map, const void *d_q, const void *d_hi,
                         uint64_t nq, void *out_q, uint32_t *pos, const BucketPlan &bp,
                         cudaStream_t s);
// Counts (and lower bounds) of the ranges from the bounds' ranks.
bt_status launch_range_gather(const bt_tree *t, const uint32_t *rank, const uint32_t *pos,
                              const void *d_lo, const void *d_hi, uint64_t nr, uint64_t *d_counts,
                              uint64_t *d_lb, cudaStream_t s);
// d_out[i] = res[pos[i]], and the found flags when d_found is not null.
bt_status launch_bucket_gather(int val_bytes, const void *res, const uint8_t *rfound,
                               const uint32_t *pos, uint64_t nq, void *d_out, uint8_t *d_found,
                               cudaStream_t s);
// Queries that a bucket search orders at a time.  A larger batch goes in equal
// parts of this many to twice this many, so that its scratch is bounded (20 bytes
// a query for 8-byte keys and values).  Larger parts gain nothing, their scattered
// passes having left the L2; smaller ones stage the tree's separators more often,
// so a tree of over 2^26 leaf blocks takes half as many queries as it has blocks.
// In one part / in parts of 2^25 (ms): 2^27 queries, 2^24 u32 keys 3.39 / 2.59;
// in parts of 2^25 / 2^24: 2^25 bounds, 2^27 u64 keys 1.01 / 1.30.
constexpr uint64_t kBucketBatch = 1ull << 25;
inline uint64_t bucket_least(const bt_tree *t) {
    return std::max<uint64_t>(kBucketBatch, t->n_sectors / 2);
}
inline uint64_t bucket_batch(const bt_tree *t, uint64_t nq) {
    const uint64_t parts = std::max<uint64_t>(1, nq / bucket_least(t));
    return (nq + parts - 1) / parts;
}
// Workspace of a bucket search: the ordered queries, every query's slot, the
// results by slot (and their found flags), the plan.
struct BucketWs {
    WsGuard ws;
    unsigned char *q = nullptr, *res = nullptr;
    uint32_t *pos = nullptr;
    uint8_t *found = nullptr;
    uint64_t max_items = 0;
    BucketPlan bp;
    explicit BucketWs(cudaStream_t s) : ws(s) {}
    static size_t up256(size_t x) { return (x + 255) / 256 * 256; }
    static size_t bytes(uint64_t nq, uint32_t buckets, size_t key_bytes, size_t res_bytes, bool flags) {
        return up256(nq * key_bytes) + up256(nq * sizeof(uint32_t)) + up256(nq * res_bytes) +
               (flags ? up256(nq) : 0) + (buckets + nq / bucket_slice(nq)) * sizeof(uint4) +
               (3 * kMaxBuckets + 64) * sizeof(uint32_t);
    }
    bt_status alloc(uint64_t nq, uint32_t buckets, size_t key_bytes, size_t res_bytes, bool flags) {
        const size_t kb = up256(nq * key_bytes), pb = up256(nq * sizeof(uint32_t));
        const size_t rb = up256(nq * res_bytes), fb = flags ? up256(nq) : 0;
        max_items = buckets + nq / bucket_slice(nq);
        const bt_status st = ws.alloc(bytes(nq, buckets, key_bytes, res_bytes, flags));
        if (st != BT_OK) return st;
        q = ws.as<unsigned char>();
        pos = reinterpret_cast<uint32_t *>(q + kb);
        res = q + kb + pb;
        found = flags ? res + rb : nullptr;
        bp.items = reinterpret_cast<uint4 *>(res + rb + fb);
        bp.scratch = reinterpret_cast<uint32_t *>(bp.items + max_items);
        bp.first = bp.scratch + 2 * kMaxBuckets;
        bp.n_items = bp.first + kMaxBuckets + 1;
        return BT_OK;
    }
};

// The tree's map: as many buckets as kMaxBuckets allows.
__host__ __device__ inline BucketMap bucket_map(uint64_t min_key, uint64_t max_key) {
    const int span = bitlen64(max_key - min_key);
    BucketMap m;
    m.min = min_key;
    m.shift = span > 11 ? span - 11 : 0;
    m.last = (uint32_t)((max_key - min_key) >> m.shift);
    return m;
}
static_assert(kMaxBuckets == 1 << 11, "bucket_map takes 11 bits");
// Measures t->bucket_blocks into *d_blocks (zeroed by the caller); the
// tree's arrays, sizes and level offsets are set.
// Does nothing when d_unsorted (optional) has bit 0 set by then.
bt_status launch_bucket_blocks(const bt_tree *t, const unsigned int *d_unsorted, uint32_t *d_blocks,
                               cudaStream_t s);
// Whether a batch is large enough to be put into an order before the search, by
// buckets or, where those do not serve and the mode asks for it, in groups.  Below
// that the order costs more than it gives, whatever the mode asks for (2^20 point
// queries, u32 keys, 2^20 / 2^26: 36 / 47 us directly, 65 / 77 grouped first; 2^19
// ranges 50 / 66 us directly, 108 / 127 grouped first).
bool point_order_pays(const bt_tree *t, uint64_t nq);
bool range_order_pays(const bt_tree *t, uint64_t nr);
// Whether a point batch is searched by buckets, and that search (workspace
// from the pool; BT_ERR_OUT_OF_MEMORY when it cannot be had).
bool bucket_search_pays(const bt_tree *t, uint64_t nq, cudaStream_t s);
bool learned_buckets_pay(const bt_tree *t, uint64_t nq, cudaStream_t s);
bool bucket_bounds_pay(const bt_tree *t, uint64_t nr, cudaStream_t s);
bt_status launch_bucket_bounds(const bt_tree *t, const void *d_lo, const void *d_hi, uint64_t nr,
                               uint64_t *d_counts, uint64_t *d_lb, cudaStream_t s);
bt_status launch_bucket_search(const bt_tree *t, const void *d_q, uint64_t nq, void *d_out,
                               cudaStream_t s, uint8_t *d_found);

// Partition kinds for launch_partition.
enum PartitionKind { kPartPoint = 0, kPart2D = 1, kPartZ = 2, kPartRadix = 3 };
// Digit bits used by the grouping passes.
constexpr int kPointGroupBits = 8;
constexpr int kRangeGroupBits = 8;

}  // namespace bt
