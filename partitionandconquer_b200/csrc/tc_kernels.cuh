// Triangle-counting intersection kernels (sm_100a).
//
// Work decomposition ("pivot" form).  Orient every undirected edge from the
// larger id to the smaller id; with degree-descending ids this is the degree
// orientation.  Let N+(x) = N(x) & [0, x) -- the prefix of x's sorted row, of
// length dplus[x] -- and N-(x) the suffix (ids > x).  A triangle a < b < c is
// found exactly once, at pivot b and in-neighbour c in N-(b), as the element
// a of N(c) & [0, b) that is also in N+(b).  Hence
//     T = sum_b sum_{c in N-(b)} |N(c) & [0,b) & N+(b)|,
// the same number as the reference's sum over partitions of
// cnt_common_neis_less_than_merge(u, v, v, i) (src/Graph.cpp:1346-1362): both
// count every triangle once.  Every kernel processes all in-edges of a set
// of pivots, so kernels can be mixed per partition and the total stays exact.
//
// Work items are (pivot, run of in-neighbours) triples taken from a global
// counter, so hub pivots with 10^5 in-neighbours are spread over many CTAs.
//
// Pivot sets in shared memory:
//  * bitmap (CTA-wide): bit a set for a in N+(b), needs b <= capacity;
//  * mixed: a bitmap of the ids below `lo` and one of the hash values of the
//    others, whose positives are looked up in an open-addressing table (<= 256
//    keys in 512 slots); its size does not grow with the pivot's id;
//  * none: threshold merge (the reference's primitive) or binary search.
#pragma once
#include <stdint.h>

#include <type_traits>

#include "pc_internal.cuh"

namespace pc {
namespace tc {

constexpr int kTile = 16384;        // pivots per planning tile
constexpr int kChunkWarp = 256;     // in-neighbours per warp work item
constexpr int kCtaThreads = 512;    // threads per CTA of the bitmap kernels
constexpr int kHashSlots = 512;     // slots per warp-private hash table
constexpr int kHashCap = 256;       // keys of a hash table (a mixed set with more is searched)
constexpr int kWarpCtaWarps = 8;    // warps per CTA of the warp kernels
constexpr int kEcRankCap = 512;     // per-edge mode: pivot sets up to this size count by rank in shared memory
constexpr int kHubHist = 8192;      // per-vertex counting: ids below this count in shared memory

enum WarpMode { kModeMerge = 1, kModeGallop = 2 };

// A pivot and a run of its in-neighbours: adj[in0, in0 + n) of the CSR.
struct __align__(16) Item {
    uint64_t in0;
    int32_t b;
    uint32_t n;
};

// First slot of row x's counters in the per-edge mode: its place in the
// oriented copy, or in the CSR when there is none (ooff null).
__device__ __forceinline__ uint64_t slot_base(const uint32_t* __restrict__ ooff, const uint64_t* __restrict__ off,
                                              int64_t x) {
    return ooff ? 4ull * ooff[x] : off[x];
}

__device__ __forceinline__ int32_t pivot_at(const int32_t* __restrict__ plist, int64_t p) {
    return plist ? plist[p] : (int32_t)p;
}

__device__ __forceinline__ uint32_t hash_slot(int32_t a) { return ((uint32_t)a * 0x9E3779B1u) >> (32 - 9); }

// Pivot sets the bitmap kernels test prefix ids against.
//
// kPlainSet: for every a in N+(b), bit a of a shared-memory bitmap, the ids of
// a word from its top bit down, so that a test is one wrapping shift and the
// word's sign (`bit_of`).
//
// kMixedSet: bit a for the ids below `lo`; for the others bit lo + h(a), h a
// hash to kFilterLog bits, and the keys in the 512-slot hash.  The set's size no
// longer grows with the pivot's id, and nearly every high id is settled by the
// one bit, because few of them are hits (5-7 % of the prefix ids at RMAT-18
// past pivot 4096, under 2 % past 16 K); the others are looked up.  The hash
// holds the last kHashCap entries of N+(b) that are not below lo; when there
// are more, its keys are found by binary search in N+(b) itself (`ovf`), so the test
// stays exact for every pivot.  With lo = 0 every id goes through the hash.
enum SetKind { kPlainSet = 0, kMixedSet = 1 };
constexpr int kFilterLog = 13;
constexpr uint32_t kFilterWords = (1u << kFilterLog) / 32;

__device__ __forceinline__ uint32_t bit_of(const uint32_t* bm, uint32_t a) {
    return __funnelshift_l(0u, bm[a >> 5], a) >> 31;
}
__device__ __forceinline__ uint32_t filter_bit(int32_t a) { return ((uint32_t)a * 0x9E3779B1u) >> (32 - kFilterLog); }

struct SetView {
    const uint32_t* bm;
    int32_t lo;                      // kMixedSet
    const int32_t* ht;               // kHashSlots slots, -1 = empty
    const uint16_t* hpos;            // per-edge counts: the rank of each slot's key
    const int32_t* __restrict__ nb;  // N+(b) + base, np entries with the copy's padding (overflow path)
    int32_t base;
    uint32_t np;
    bool ovf;
    // the bit an id is tested at
    template <int kKind>
    __device__ __forceinline__ uint32_t place(int32_t a) const {
        if (kKind == kPlainSet) return (uint32_t)a;
        return a < lo ? (uint32_t)a : (uint32_t)lo + filter_bit(a);
    }
    // whether a is among the hash's keys, and its rank in N+(b) (hpos not null, or ovf) or its slot
    __device__ __forceinline__ bool find(int32_t a, uint32_t* rank) const {
        if (ovf) {
            uint32_t lo = 0, hi = np;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (__ldg(nb + mid) - base < a) lo = mid + 1; else hi = mid;
            }
            *rank = lo;
            return lo < np && __ldg(nb + lo) - base == a;
        }
        uint32_t s = hash_slot(a);
        for (int32_t key; (key = ht[s]) != -1; s = (s + 1) & (kHashSlots - 1))
            if (key == a) {
                *rank = hpos ? hpos[s] : s;
                return true;
            }
        return false;
    }
};

// Shared-memory words of one pivot set: the bitmap, then the hash of a mixed
// set; in the per-edge mode also a plain set's ranks (a 16-bit one per word, a
// 32-bit one per 64 words) or a mixed set's (one per slot), and the hits by
// rank; in the per-vertex mode a mixed set's hits by slot.
constexpr uint32_t kSlotRankWords = (uint32_t)kHashSlots / 2;
constexpr uint32_t bitmap_set_words(uint32_t bm_words, int mode, int kind) {
    return bm_words + (kind == kMixedSet ? (uint32_t)kHashSlots + (mode == 1 ? kSlotRankWords : 0u) : 0u) +
           (mode != 2 ? 0u
                      : (kind == kPlainSet ? (bm_words + 63) / 64 + (bm_words + 1) / 2 : kSlotRankWords) +
                            (uint32_t)kEcRankCap);
}

// Named barrier over `nthreads` threads of one warp group (ids 1..15; id 0
// is __syncthreads).
__device__ __forceinline__ void group_barrier(int id, int nthreads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

// Per-vertex triangle counts (kCountVertex): every triangle found adds 1 to its
// lowest vertex a; ids below kHubHist go to a shared-memory histogram
// (almost every hit is a hub), the rest to the global counts.
__device__ __forceinline__ void count_vertex(int32_t a, unsigned long long* __restrict__ tri, uint32_t* hist,
                                             int32_t hist_ids = kHubHist) {
    if (a < hist_ids) atomicAdd(&hist[a], 1u);
    else atomicAdd(&tri[a], 1ull);
}

// What the pivot-form kernels count: triangles; per-vertex triangle counts
// (LCC); per-edge counts at the oriented slots (Jaccard), where every
// triangle a < b < c adds 1 to the slot of a in row c (its scan index), to the
// slot of a in row b (its rank in the pivot set) and, once per pair, its
// hits to the slot of b in row c (where the scan stops).  The slot of edge
// {x, y}, y < x, is the position of y in row x of the oriented copy.
enum CountMode { kCountOnly = 0, kCountVertex = 1, kCountEdge = 2 };

// The rows N+(x) that the set kernels scan.
//
// OrientedView is the oriented copy (build_oriented): row x holds N+(x) in
// ascending order, starts at 16-byte vector off[x] of ids and is padded with
// INT_MAX to whole vectors; at least 32 vectors of INT_MAX follow the last row.
//
// CsrView is the CSR itself, for graphs whose copy has no room: the vectors that
// hold a row begin up to 3 ids before it and end after it, so every id's place is
// compared with the row's bounds.  With groups of 4 lanes only.
struct OrientedView {
    static constexpr bool kCsr = false;
    using Pos = uint32_t;
    const uint32_t* __restrict__ off;
    const int4* __restrict__ ids;
    // a row as a pivot set: n vectors from v0, the k-th of them, the id before
    // it, all as a sorted array, and the slot of the first id
    struct Row {
        uint32_t v0, n;
    };
    __device__ __forceinline__ Row row(int32_t b) const { return Row{off[b], off[b + 1] - off[b]}; }
    __device__ __forceinline__ int4 vector(const Row& r, uint32_t k) const { return __ldg(ids + (r.v0 + k)); }
    __device__ __forceinline__ int32_t before(const Row& r, uint32_t k) const { return __ldg(&ids[r.v0 + k - 1].w); }
    __device__ __forceinline__ void sorted(const Row& r, SetView* S) const {
        S->nb = reinterpret_cast<const int32_t*>(ids + r.v0);
        S->np = 4 * r.n;
        S->base = 0;
    }
    __device__ __forceinline__ uint64_t slot(const Row& r) const { return 4ull * r.v0; }
};

struct CsrView {
    static constexpr bool kCsr = true;
    using Pos = uint64_t;
    const uint64_t* __restrict__ off;
    const int32_t* __restrict__ adj;
    const uint32_t* __restrict__ dplus;
    int32_t base;  // subtracted from the ids
    struct Row {
        uint64_t e0;
        uint32_t n, len;  // n vectors for len entries
    };
    __device__ __forceinline__ Row row(int32_t b) const { return Row{off[b], (dplus[b] + 3) / 4, dplus[b]}; }
    __device__ __forceinline__ int4 vector(const Row& r, uint32_t k) const {
        const int32_t* p = adj + r.e0 + 4ull * k;
        const uint32_t left = r.len - 4 * k;
        int4 v = make_int4(__ldg(p) - base, INT32_MAX, INT32_MAX, INT32_MAX);
        if (left > 1) v.y = __ldg(p + 1) - base;
        if (left > 2) v.z = __ldg(p + 2) - base;
        if (left > 3) v.w = __ldg(p + 3) - base;
        return v;
    }
    __device__ __forceinline__ int32_t before(const Row& r, uint32_t k) const {
        return __ldg(adj + r.e0 + 4ull * k - 1) - base;
    }
    __device__ __forceinline__ void sorted(const Row& r, SetView* S) const {
        S->nb = adj + r.e0;
        S->np = r.len;
        S->base = base;
    }
    __device__ __forceinline__ uint64_t slot(const Row& r) const { return r.e0; }
};

// Ranks in a pivot set (per-edge counts): r16[w] is the rank, modulo 2^16, of
// the first entry with its bit in word w, and r32[w / 64] that of the first
// entry of the 64-word block; words without entries hold old values.
struct SetRanks {
    const uint16_t* r16;
    const uint32_t* r32;
};
__device__ __forceinline__ uint32_t rank_in_set(const uint32_t* bm, const SetRanks& R, int32_t a) {
    const uint32_t w = (uint32_t)a >> 5, base = R.r32[w >> 6];
    return base + (uint16_t)(R.r16[w] - (uint16_t)base) + __popc(__funnelshift_rc(bm[w], 0u, 32u - ((uint32_t)a & 31u)));
}

// Where the hits of one warp's scans go besides the count.
struct HitSink {
    unsigned long long* __restrict__ tri;  // kCountVertex: per-vertex counts, of in-neighbours
    unsigned long long* tri_low;           // ... and of the ids in the oriented copy
    uint32_t* hist;                        // ... whose first hist_ids ids count here
    int32_t hist_ids;
    uint32_t* by_slot;                     // ... of a mixed set's hash: 16-bit counters, or null
    uint32_t* used;                        // ... set with the first of them
    uint32_t* __restrict__ ecnt;           // kCountEdge: per-slot counts
    uint32_t* by_rank;                     // ... of row b: shared counters, or its slots in ecnt
    SetRanks ranks;
};

// Scans the prefixes of up to 32 in-neighbours of pivot b: lane j < nb holds
// in-neighbour j's id (c); returns this lane's hits.
//
// A group of G lanes takes one in-neighbour at a time, V vectors of 4 ids per
// lane and step, and goes on to its next one (NG apart) as soon as its row reaches an
// id >= b (b itself, which a symmetric adjacency has in the row, or the INT_MAX
// at an unchecked row's end: a scan ends inside its row), while the
// other groups go on with theirs: no lane waits for the longest of the 32 / G
// rows in flight.  All groups step together, so the vote that ends a row is
// one full-warp ballot, and the load of the next vector is issued between
// that vote and the tests of the current ids: it is never speculative.
// Nothing is checked per id: ids past the end of the row (the lanes behind
// the stop, then a running maximum inside the stopping vector) become >= b,
// and min(id, b) sends them all to b, whose bit is never set (in a mixed set
// it may be another key's bit; the look-up settles that).
//
// Bound: shared-memory wavefronts and instruction issue (RMAT-20's plain sets: L1
// at 95 %, 80 % of the issue slots, 32 of 32 lanes active), then L2 latency.  About 45
// warp instructions per 128 ids; the earlier scan, which tested each id's
// position and kept a group waiting for the longest of its warp's rows, took
// about 130.  Bitmap kernels of RMAT-20: 2.07 -> 0.83 ms; RMAT-24's unit of ids
// 49-65 K (2.0e9 ids): 3.23 -> 1.92 ms with G = 8 and V = 1.
//
// Two vectors a step keep twice the bytes in flight and halve the votes per id
// where prefixes are long; short ones waste the second.  RMAT-24 by (G, V), ms:
// that unit (8, 1) 1.95, (4, 1) 2.05, (4, 2) 1.82, (8, 2) 1.65, (2, 2) 2.21; the
// first unit's tail with its matrix part 8.3 / 8.0 / 7.4 / 8.4 / 7.0; RMAT-20's
// light pivots, ER-20: 0.98 / 0.83 / 1.01 / 1.41 / 0.95.  So bitmap sets scan with
// (4, 2), light pivots with (4, 1).
//
// On the CSR (CsrView) a step also masks the ids outside the row, and rows start
// anywhere in a sector: counts of RMAT-24 / 22 / 20 / 16 take 35.0 / 6.2 / 1.83 /
// 0.16 ms, on the copy 24.9 / 4.3 / 0.99 / 0.12.
template <int G, int V, int kMode, int kKind, class Rows>
__device__ __forceinline__ uint32_t scan_in_neighbours(const Rows& R, int32_t c, int nb, int32_t b, const SetView& S,
                                                       int lane, const HitSink& sink) {
    constexpr bool kCsr = Rows::kCsr;
    using Pos = typename Rows::Pos;
    static_assert(!kCsr || G == 4, "scans of the CSR take groups of 4 lanes");
    constexpr int NG = 32 / G;
    const int gl = lane % G;
    const unsigned gmask = G == 32 ? 0xffffffffu : (((1u << G) - 1u) << (lane & ~(G - 1)));
    const unsigned below = gmask & ((1u << lane) - 1u);
    const int4 none = make_int4(INT32_MAX, INT32_MAX, INT32_MAX, INT32_MAX);
    int j = lane / G;
    // the row starts: vectors of the copy, entries of the CSR (with the rows' lengths)
    const Pos start = R.off[c];
    uint32_t len = 0;
    if constexpr (kCsr) len = R.dplus[c];
    Pos e0 = __shfl_sync(0xffffffffu, start, j), e1 = 0;  // CSR: the current row's entries are [e0, e1)
    Pos q = (kCsr ? e0 / 4 : e0) + gl;
    if constexpr (kCsr) e1 = e0 + __shfl_sync(0xffffffffu, len, j);
    bool act = j < nb;
    int4 v[V];
    auto load = [&](int i) {
        if constexpr (kCsr) return act && 4 * (q + i * G) < e1 ? __ldg(reinterpret_cast<const int4*>(R.adj) + q + i * G) : none;
        // (the sum in 32 bits suits the count's registers, not the other modes':
        // RMAT-20's plain sets 698 and 731 us, per vertex 1220 and 1205)
        else if constexpr (kMode == kCountOnly) return act ? __ldg(R.ids + (q + i * G)) : none;
        else return act ? __ldg(R.ids + q + i * G) : none;
    };
#pragma unroll
    for (int i = 0; i < V; ++i) v[i] = load(i);
    uint32_t cnt = 0, pair = 0;
    while (__any_sync(0xffffffffu, act)) {
        // CSR: ids before the row become the smallest id, those after it the
        // largest; lead ids of the vector are before it (0 to 3)
        int lead[kCsr ? V : 1];
        if constexpr (kCsr) {
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const Pos p = 4 * (q + i * G);
                lead[i] = act && p < e0 ? (int)(e0 - p) : 0;
                const int end = act && p < e1 ? (int)min(e1 - p, (Pos)4) : 0;
                v[i].x = lead[i] > 0 ? INT32_MIN : (end > 0 ? v[i].x - R.base : INT32_MAX);
                v[i].y = lead[i] > 1 ? INT32_MIN : (end > 1 ? v[i].y - R.base : INT32_MAX);
                v[i].z = lead[i] > 2 ? INT32_MIN : (end > 2 ? v[i].z - R.base : INT32_MAX);
                v[i].w = end > 3 ? v[i].w - R.base : INT32_MAX;
            }
        }
        // vector i of the group's lanes precedes vector i + 1: the row's stop is
        // the lowest lane of the first vector that has one
        unsigned stop[V];
        bool past[V];  // this lane's vector lies behind the stop
        bool done = false;
        int4 a[V];
#pragma unroll
        for (int i = 0; i < V; ++i) {
            stop[i] = __ballot_sync(0xffffffffu, v[i].w >= b);
            past[i] = done || (G > 1 && (stop[i] & below) != 0);
            done = done || (G == 1 ? v[i].w >= b : (stop[i] & gmask) != 0);
            a[i] = v[i];
            if (past[i]) a[i].x = INT32_MAX;
        }
        const Pos qc = q;
        const int jc = j;
        if (done) j += NG;
        const Pos s = __shfl_sync(0xffffffffu, start, j & 31);
        q = done ? (kCsr ? s / 4 : s) + gl : q + V * G;
        if constexpr (kCsr) {
            const uint32_t l = __shfl_sync(0xffffffffu, len, j & 31);
            if (done) {
                e0 = s;
                e1 = s + l;
            }
        }
        const bool had = act;
        act = j < nb;
#pragma unroll
        for (int i = 0; i < V; ++i) v[i] = load(i);
        uint32_t hits = 0;
#pragma unroll
        for (int i = 0; i < V; ++i) {
            a[i].y = max(a[i].x, a[i].y);
            a[i].z = max(a[i].y, a[i].z);
            a[i].w = max(a[i].z, a[i].w);
            int32_t e[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
            if constexpr (kCsr) {
#pragma unroll
                for (int t = 0; t < 3; ++t)
                    if (t < lead[i]) e[t] = INT32_MAX;
            }
            uint32_t h[4];
            uint32_t rank[4];  // kMixedSet: of the hits at or past lo
#pragma unroll
            for (int t = 0; t < 4; ++t) h[t] = bit_of(S.bm, S.place<kKind>(min(e[t], b)));
            if constexpr (kKind == kMixedSet) {
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (h[t] && e[t] >= S.lo) h[t] = e[t] < b && S.find(e[t], &rank[t]);
            }
            const uint32_t here = h[0] + h[1] + h[2] + h[3];
            hits += here;
            if constexpr (kMode != kCountOnly) {
                if (here) {
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        if (!h[t]) continue;
                        if constexpr (kMode == kCountVertex) {
                            if (e[t] < sink.hist_ids) {
                                atomicAdd(&sink.hist[e[t]], 1u);
                            } else if (kKind == kMixedSet && sink.by_slot && e[t] >= S.lo && !S.ovf) {
                                atomicAdd(sink.by_slot + (rank[t] >> 1), 1u << (16 * (rank[t] & 1)));
                                *sink.used = 1;
                            } else {
                                atomicAdd(&sink.tri_low[e[t]], 1ull);
                            }
                        } else {
                            atomicAdd(sink.ecnt + (4ull * (qc + i * G) + t), 1u);
                            atomicAdd(sink.by_rank +
                                          (kKind == kMixedSet ? rank[t] : rank_in_set(S.bm, sink.ranks, e[t])),
                                      1u);
                        }
                    }
                }
            }
        }
        cnt += hits;
        if constexpr (kMode != kCountOnly) {
            pair += hits;
            if (__any_sync(0xffffffffu, done && had)) {
                uint32_t sum = pair;
                for (int o = G / 2; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                if constexpr (kMode == kCountVertex) {
                    const int32_t cj = __shfl_sync(0xffffffffu, c, jc & 31);
                    if (done && had && gl == 0 && sum) atomicAdd(&sink.tri[cj], (unsigned long long)sum);
                } else {
                    // the stop holds b: after the ids below it
#pragma unroll
                    for (int i = 0; i < V; ++i)
                        if (done && had && sum && ((stop[i] >> lane) & 1u) && !past[i])
                            atomicAdd(sink.ecnt + (4ull * (qc + i * G) + (a[i].x < b) + (a[i].y < b) + (a[i].z < b)), sum);
                }
                if (done) pair = 0;
            }
        }
    }
    return cnt;
}

// CTAs per SM a bitmap kernel's registers leave room for.  Three for the count;
// two for split sets with two vectors a step, whose look-ups spill at 40
// registers (RMAT-24's unit of ids 65-82 K: 1.10 ms, 1.28 with three), for scans of
// the CSR with two vectors a step, which spill too, and for the other modes.
constexpr int bitmap_ctas(int V, int mode, int kind, bool csr) {
    return mode == kCountOnly && !((kind == kMixedSet || csr) && V > 1) ? 3 : 2;
}

// Bitmap kernel: a CTA of kCtaThreads threads holds 16/K pivot sets in
// shared memory, one per group of K warps; each group takes its own work
// items (pivot, a run of its in-neighbours), so a group synchronises only
// with itself (a named barrier, or nothing when K == 1).  A warp fetches 32
// in-neighbours' ids with one coalesced load and their row starts with 32
// independent gathers and scans their prefixes (scan_in_neighbours).
// Mixed sets have (bm_words - kFilterWords) * 32 = lo bits for the low ids,
// whatever the pivots' ids (0 in the per-edge mode, which needs every hit's
// rank).
template <int K, int G, int V, int kMode, int kKind, class Rows>
__global__ void __launch_bounds__(kCtaThreads, bitmap_ctas(V, kMode, kKind, Rows::kCsr))
    k_tc_bitmap(Rows R, const int32_t* __restrict__ adj, const Item* __restrict__ items,
                const uint32_t* __restrict__ nitems_p, uint32_t cap, uint32_t* __restrict__ next_item,
                unsigned long long* __restrict__ total, uint32_t bm_words, unsigned long long* __restrict__ unit_cost,
                const int32_t* __restrict__ unit_of, unsigned long long* __restrict__ tri,
                uint32_t* __restrict__ ecnt) {
    constexpr bool kHash = kKind == kMixedSet;
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t s_item[16];
    __shared__ uint32_t s_used[16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int set = warp / K, wi = warp % K;
    constexpr int nsets = (kCtaThreads / 32) / K;
    constexpr int set_threads = K * 32;
    const int tis = wi * 32 + lane;
    const uint32_t set_words = bitmap_set_words(bm_words, kMode, kKind);
    uint32_t* bm = smem + (size_t)set * set_words;
    int32_t* ht = reinterpret_cast<int32_t*>(bm + bm_words);  // kHash: the set's hash slots
    // kCountEdge: a plain set's ranks, or the rank of each hash slot's key; kCountVertex:
    // the hits of each hash slot's key (an item has at most kCtaThreads / 2 in-neighbours)
    uint32_t* r32 = bm + bm_words + (kHash ? (uint32_t)kHashSlots : 0u);
    uint16_t* r16 = reinterpret_cast<uint16_t*>(r32 + (kHash ? 0u : (bm_words + 63) / 64));
    uint32_t* by_rank = bm + set_words - kEcRankCap;
    uint32_t* hist = smem + (size_t)nsets * set_words;        // kCountVertex: kHubHist counters after the sets
    for (uint32_t i = tis; i < set_words; i += set_threads) bm[i] = 0;
    if (kHash)
        for (uint32_t i = tis; i < (uint32_t)kHashSlots; i += set_threads) ht[i] = -1;
    if (kMode == kCountVertex)
        for (uint32_t i = tid; i < (uint32_t)kHubHist; i += blockDim.x) hist[i] = 0;
    if (tid < 16) s_used[tid] = 0;
    __syncthreads();
    auto set_sync = [&]() {
        if constexpr (K == 1) __syncwarp();
        else group_barrier(1 + set, set_threads);
    };
    const int32_t lo = kHash ? (int32_t)(bm_words - kFilterWords) * 32 : 0;
    const uint32_t nitems = min(*nitems_p, cap);
    unsigned long long cnt = 0;
    for (;;) {
        if (tis == 0) s_item[set] = atomicAdd(next_item, 1u);
        set_sync();
        const uint32_t it = s_item[set];
        if (it >= nitems) break;
        const long long t0 = unit_cost ? clock64() : 0;
        const Item I = items[it];
        const int32_t b = I.b;
        const typename Rows::Row row = R.row(b);
        SetView S;
        S.bm = bm;
        S.lo = lo;
        S.ht = ht;
        S.hpos = kHash && kMode == kCountEdge ? r16 : nullptr;
        R.sorted(row, &S);
        // the hash takes ranks np - kHashCap and up: all high ids, or it is not used
        S.ovf = kHash && S.np > (uint32_t)kHashCap && __ldg(S.nb + (S.np - kHashCap - 1)) - S.base >= lo;
        for (uint32_t k = tis; k < row.n; k += set_threads) {
            const int4 v = R.vector(row, k);
            const int32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int32_t a = e[t];
                if (a == INT32_MAX) continue;  // padding
                const uint32_t rank = 4 * k + t;
                const uint32_t x = S.place<kKind>(a);
                atomicOr(&bm[x >> 5], 0x80000000u >> (x & 31));
                if (kHash && !S.ovf && a >= lo) {
                    // at most kHashCap keys in kHashSlots slots: a free slot exists
                    uint32_t hs = hash_slot(a);
                    while (atomicCAS(&ht[hs], -1, a) != -1) hs = (hs + 1) & (kHashSlots - 1);
                    if (kMode == kCountEdge) r16[hs] = (uint16_t)rank;
                }
                if (kMode == kCountEdge && kKind == kPlainSet) {
                    const int32_t prev = t ? e[t - 1] : (k ? R.before(row, k) : -1);
                    if (prev < 0 || (prev >> 5) != (a >> 5)) r16[a >> 5] = (uint16_t)rank;
                    if (prev < 0 || (prev >> 11) != (a >> 11)) r32[a >> 11] = rank;
                }
            }
        }
        set_sync();
        const bool few = S.np <= (uint32_t)kEcRankCap;
        HitSink sink;
        sink.tri = sink.tri_low = tri;
        sink.hist = hist;
        sink.hist_ids = kHubHist;
        sink.by_slot = kHash && kMode == kCountVertex ? r32 : nullptr;
        sink.used = s_used + set;
        sink.ecnt = ecnt;
        sink.by_rank = few ? by_rank : ecnt + R.slot(row);
        sink.ranks = SetRanks{r16, r32};
        const unsigned long long cnt0 = cnt;
        for (uint32_t k = wi * 32; k < I.n; k += set_threads) {
            const int nb = min(32, (int)(I.n - k));
            const int32_t c = lane < nb ? adj[I.in0 + k + lane] : 0;
            cnt += scan_in_neighbours<G, V, kMode, kKind>(R, c, nb, b, S, lane, sink);
        }
        if (kMode == kCountVertex) {
            unsigned long long hb = cnt - cnt0;  // this item's triangles at pivot b
            for (int o = 16; o; o >>= 1) hb += __shfl_xor_sync(0xffffffffu, hb, o);
            if (lane == 0 && hb) atomicAdd(&tri[b], hb);
            if (kHash) {
                // the hits of the hash's keys, eight counters a load.  (One global
                // atomic for each of them took 4000 cliques of 64 vertices 3.2 ms a
                // call, counted by slot first 0.84; RMAT-16 0.189 and 0.193.)
                set_sync();
                const bool used = s_used[set];
                set_sync();  // all have read it
                if (used) {
                    if (tis == 0) s_used[set] = 0;
                    uint4* c4 = reinterpret_cast<uint4*>(r32);
                    for (uint32_t x = tis; x < (uint32_t)kHashSlots / 8; x += set_threads) {
                        const uint4 c = c4[x];
                        if (!(c.x | c.y | c.z | c.w)) continue;
                        c4[x] = make_uint4(0, 0, 0, 0);
                        const uint32_t w[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
                        for (int t = 0; t < 8; ++t) {
                            const uint32_t h = w[t / 2] >> (16 * (t & 1)) & 0xffffu;
                            if (h) atomicAdd(&tri[ht[8 * x + t]], (unsigned long long)h);
                        }
                    }
                }
            }
        }
        set_sync();
        for (uint32_t k = tis; k < row.n; k += set_threads) {
            const int4 v = R.vector(row, k);
            const int32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                if (kHash || e[t] != INT32_MAX) bm[S.place<kKind>(e[t]) >> 5] = 0;
                if (kMode == kCountEdge && few) {
                    const uint32_t h = by_rank[4 * k + t];
                    if (h) {
                        atomicAdd(ecnt + (R.slot(row) + 4 * k + t), h);
                        by_rank[4 * k + t] = 0;
                    }
                }
            }
        }
        if (kHash && !S.ovf)
            for (uint32_t x = tis; x < (uint32_t)kHashSlots; x += set_threads) ht[x] = -1;
        set_sync();
        // profiling runs: the set's warp-cycles on this item, charged to its unit
        if (unit_cost && tis == 0) atomicAdd(&unit_cost[unit_of[b]], (unsigned long long)(clock64() - t0) * K);
    }
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0 && cnt) atomicAdd(total, cnt);
    if (kMode == kCountVertex) {
        __syncthreads();
        for (uint32_t i = tid; i < (uint32_t)kHubHist; i += blockDim.x)
            if (hist[i]) atomicAdd(&tri[i], (unsigned long long)hist[i]);
    }
}

// |x & y & [0, thr)| for sorted x, y: Partitioned_Graph::
// cnt_common_neis_less_than_merge (src/Graph.cpp:1132-1153), without its
// one-past-the-end reads.
__device__ __forceinline__ uint32_t merge_below(const int32_t* __restrict__ x, uint32_t nx,
                                                const int32_t* __restrict__ y, uint32_t ny, int32_t thr) {
    uint32_t i = 0, j = 0, c = 0;
    while (i < nx && j < ny) {
        const int32_t a = x[i], bb = y[j];
        if (a >= thr || bb >= thr) break;
        if (a < bb) ++i;
        else if (a > bb) ++j;
        else { ++c; ++i; ++j; }
    }
    return c;
}

// Each id of N(c) & [0, thr) looked up in N+(b) by binary search: the
// lower_bound probing of Partitioned_Graph::cnt_common_neis_galloping
// (src/Graph.cpp:1071-1085).
__device__ __forceinline__ uint32_t gallop_below(const int32_t* __restrict__ x, uint32_t nx,
                                                 const int32_t* __restrict__ y, uint32_t ny, int32_t thr) {
    uint32_t c = 0;
    for (uint32_t i = 0; i < nx; ++i) {
        const int32_t a = x[i];
        if (a >= thr) break;
        uint32_t lo = 0, hi = ny;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (y[mid] < a) lo = mid + 1; else hi = mid;
        }
        c += (lo < ny && y[lo] == a) ? 1u : 0u;
    }
    return c;
}

// merge_below / gallop_below with per-vertex counting of every match (kVC).
template <bool kVC>
__device__ __forceinline__ uint32_t merge_below_vc(const int32_t* __restrict__ x, uint32_t nx,
                                                   const int32_t* __restrict__ y, uint32_t ny, int32_t thr,
                                                   unsigned long long* __restrict__ tri, uint32_t* hist) {
    uint32_t i = 0, j = 0, c = 0;
    while (i < nx && j < ny) {
        const int32_t a = x[i], bb = y[j];
        if (a >= thr || bb >= thr) break;
        if (a < bb) ++i;
        else if (a > bb) ++j;
        else {
            ++c;
            if (kVC) count_vertex(a, tri, hist);
            ++i;
            ++j;
        }
    }
    return c;
}

template <bool kVC>
__device__ __forceinline__ uint32_t gallop_below_vc(const int32_t* __restrict__ x, uint32_t nx,
                                                    const int32_t* __restrict__ y, uint32_t ny, int32_t thr,
                                                    unsigned long long* __restrict__ tri, uint32_t* hist) {
    uint32_t c = 0;
    for (uint32_t i = 0; i < nx; ++i) {
        const int32_t a = x[i];
        if (a >= thr) break;
        uint32_t lo = 0, hi = ny;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (y[mid] < a) lo = mid + 1; else hi = mid;
        }
        if (lo < ny && y[lo] == a) {
            ++c;
            if (kVC) count_vertex(a, tri, hist);
        }
    }
    return c;
}

// Per-edge forms (kEC): matches add 1 to the slots of a in row c (x) and in
// the pivot set (y); the pair's total goes to the slot of b = thr in x.
__device__ __forceinline__ uint32_t merge_below_ec(const int32_t* __restrict__ x, uint32_t nx,
                                                   const int32_t* __restrict__ y, uint32_t ny, int32_t thr,
                                                   uint32_t* __restrict__ ec_x, uint32_t* __restrict__ ec_y) {
    uint32_t i = 0, j = 0, c = 0;
    while (i < nx && j < ny) {
        const int32_t a = x[i], bb = y[j];
        if (a >= thr || bb >= thr) break;
        if (a < bb) ++i;
        else if (a > bb) ++j;
        else {
            ++c;
            atomicAdd(&ec_x[i], 1u);
            atomicAdd(&ec_y[j], 1u);
            ++i;
            ++j;
        }
    }
    while (i < nx && x[i] < thr) ++i;
    if (c && i < nx) atomicAdd(&ec_x[i], c);  // x[i] == thr: thr is in x
    return c;
}

__device__ __forceinline__ uint32_t gallop_below_ec(const int32_t* __restrict__ x, uint32_t nx,
                                                    const int32_t* __restrict__ y, uint32_t ny, int32_t thr,
                                                    uint32_t* __restrict__ ec_x, uint32_t* __restrict__ ec_y) {
    uint32_t c = 0, i = 0;
    for (; i < nx; ++i) {
        const int32_t a = x[i];
        if (a >= thr) break;
        uint32_t lo = 0, hi = ny;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (y[mid] < a) lo = mid + 1; else hi = mid;
        }
        if (lo < ny && y[lo] == a) {
            ++c;
            atomicAdd(&ec_x[i], 1u);
            atomicAdd(&ec_y[lo], 1u);
        }
    }
    if (c && i < nx) atomicAdd(&ec_x[i], c);
    return c;
}

// Warp kernels: one item (pivot, <= kChunkWarp in-neighbours) per warp, one
// lane per in-neighbour.
template <int MODE, bool kVC = false, bool kEC = false>
__global__ void __launch_bounds__(kWarpCtaWarps * 32) k_tc_warp(const uint64_t* __restrict__ off,
                                                                const int32_t* __restrict__ adj,
                                                                const uint32_t* __restrict__ dplus,
                                                                const uint32_t* __restrict__ ooff,
                                                                const Item* __restrict__ items,
                                                                const uint32_t* __restrict__ nitems_p,
                                                                uint32_t cap,
                                                                uint32_t* __restrict__ next_item,
                                                                unsigned long long* __restrict__ total,
                                                                unsigned long long* __restrict__ unit_cost,
                                                                const int32_t* __restrict__ unit_of,
                                                                unsigned long long* __restrict__ tri,
                                                                uint32_t* __restrict__ ecnt) {
    __shared__ uint32_t hist[kVC ? kHubHist : 1];
    const int lane = threadIdx.x & 31;
    if (kVC) {
        for (int i = threadIdx.x; i < kHubHist; i += blockDim.x) hist[i] = 0;
        __syncthreads();
    }
    const uint32_t nitems = min(*nitems_p, cap);
    unsigned long long cnt = 0;
    for (;;) {
        uint32_t it = 0;
        if (lane == 0) it = atomicAdd(next_item, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= nitems) break;
        const long long t0 = unit_cost ? clock64() : 0;
        const unsigned long long cnt_item0 = cnt;
        const Item I = items[it];
        const int32_t b = I.b;
        const uint64_t rb = off[b];
        const uint32_t dp = dplus[b];
        const uint64_t in0 = I.in0, in1 = I.in0 + I.n;
        const int32_t* nb = adj + rb;
        uint32_t* eb = kEC ? ecnt + slot_base(ooff, off, b) : nullptr;
        if (MODE == kModeGallop) {
            for (uint64_t e = in0 + lane; e < in1; e += 32) {
                const int32_t c = adj[e];
                if (kEC) {
                    cnt += gallop_below_ec(adj + off[c], dplus[c], nb, dp, b, ecnt + slot_base(ooff, off, c), eb);
                    continue;
                }
                const uint32_t h = gallop_below_vc<kVC>(adj + off[c], dplus[c], nb, dp, b, tri, hist);
                cnt += h;
                if (kVC && h) atomicAdd(&tri[c], (unsigned long long)h);
            }
        } else {
            for (uint64_t e = in0 + lane; e < in1; e += 32) {
                const int32_t c = adj[e];
                if (kEC) {
                    cnt += merge_below_ec(adj + off[c], dplus[c], nb, dp, b, ecnt + slot_base(ooff, off, c), eb);
                    continue;
                }
                const uint32_t h = merge_below_vc<kVC>(adj + off[c], dplus[c], nb, dp, b, tri, hist);
                cnt += h;
                if (kVC && h) atomicAdd(&tri[c], (unsigned long long)h);
            }
        }
        if (unit_cost) {
            __syncwarp();
            if (lane == 0) atomicAdd(&unit_cost[unit_of[b]], (unsigned long long)(clock64() - t0));
        }
        if (kVC) {
            // this item's triangles at pivot b: the warp's hits since the item began
            unsigned long long hb = cnt - cnt_item0;
            for (int o = 16; o; o >>= 1) hb += __shfl_xor_sync(0xffffffffu, hb, o);
            if (lane == 0 && hb) atomicAdd(&tri[b], hb);
        }
    }
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0 && cnt) atomicAdd(total, cnt);
    if (kVC) {
        __syncthreads();
        for (int i = threadIdx.x; i < kHubHist; i += blockDim.x)
            if (hist[i]) atomicAdd(&tri[i], (unsigned long long)hist[i]);
    }
}


// ---- in-neighbour-major form for hub units (variant "matrix") ----------------
//
// For a unit of pivots b in the id range [lo, hi) (hi <= kMatrixMaxId), the
// pivot sets N+(b) are kept as bitmap rows H[b - lo] of hi bits in global
// memory: (hi - lo) * hi / 8 bytes, 32 MB for the first 16 K ids, which stay
// in L2.  The kernel then walks the in-neighbours c instead of the pivots:
// S_c = N(c) & [0, min(hi, c)) is read once, and for every pivot b in
// S_c & [lo, hi) at position j of S_c the count |S_c[0..j) & N+(b)| is taken
// either by j bit probes into H[b] or by ceil(b/32) word-wise ANDs of H[b]
// with a shared-memory bitmap of S_c and popcounts, whichever is cheaper.
// Every (pivot, in-neighbour) pair of the unit is one pair (b, c) here, so the
// count equals the pivot form's; what changes is that N(c) is read once per c
// instead of once per pivot.  Only the hubs' pairs run this way (kMatrixFrom in
// tc.cu); the other in-neighbours of the unit are items of the bitmap kernels.
constexpr int kMatrixMaxId = 1 << 16;      // hi bound: rows of <= 8 KB (H: kMatrixRowsCap in tc.cu)
constexpr int kMatrixWarps = 8;            // warps per CTA
constexpr int kMatrixBlock = 8;            // pivots a warp takes at a time

__device__ __forceinline__ uint32_t lower_bound_i32(const int32_t* __restrict__ p, uint32_t n, int32_t x) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (p[mid] < x) lo = mid + 1; else hi = mid;
    }
    return lo;
}

}  // namespace tc
}  // namespace pc
