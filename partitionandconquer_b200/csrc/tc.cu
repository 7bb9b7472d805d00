// Triangle counting: planning units, per-unit features, variant selection
// (forced / heuristic / learned) and the pc_tc entry points.
#include <algorithm>
#include <initializer_list>
#include <cmath>
#include <cstring>

#include "selector.cuh"
#include "tc_kernels.cuh"

namespace pc {
namespace tc {

// ---- planning units ----------------------------------------------------------
// A unit is a run of <= kTile consecutive plist positions inside one
// partition: partitions are the planning granularity, and oversized
// partitions (and the single partition of an unpartitioned graph) are split
// into tiles.

static void build_units(const pc_pgraph* pg, std::vector<int64_t>* lo, std::vector<int64_t>* hi) {
    lo->clear();
    hi->clear();
    for (int k = 0; k < pg->P; ++k) {
        for (int64_t p = pg->pstart[k]; p < pg->pstart[k + 1]; p += kTile) {
            lo->push_back(p);
            hi->push_back(std::min<int64_t>(p + kTile, pg->pstart[k + 1]));
        }
    }
}

// Unit of every pivot (plist position ranges -> vertex ids).
__global__ void k_unit_of(const int32_t* __restrict__ plist, const int64_t* __restrict__ lo,
                          const int64_t* __restrict__ hi, int32_t* __restrict__ unit_of) {
    const int64_t p0 = lo[blockIdx.x], p1 = hi[blockIdx.x];
    for (int64_t p = p0 + threadIdx.x; p < p1; p += blockDim.x) unit_of[pivot_at(plist, p)] = (int32_t)blockIdx.x;
}

// Per-pivot statistics, one thread per vertex; when a whole warp lies in one
// unit (the common case: units are runs of positions) it reduces first and
// lane 0 issues the atomics.
__global__ void k_unit_pivot_stats(const uint64_t* __restrict__ off, const uint32_t* __restrict__ dplus,
                                   const int32_t* __restrict__ unit_of, uint64_t n,
                                   unsigned long long* __restrict__ out /* kRawStats per unit */) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t nr = (n + 31) & ~31ull;
    const int lane = threadIdx.x & 31;
    for (uint64_t b = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; b < nr; b += stride) {
        const bool ok = b < n;
        int32_t u = -1;
        unsigned long long v[7] = {0, 0, 0, 0, 0, 0, 0};
        if (ok) {
            u = unit_of[b];
            const uint64_t deg = off[b + 1] - off[b];
            const uint32_t dp = dplus[b];
            const double ld = log2(1.0 + (double)deg);
            v[0] = 1;
            v[1] = deg - dp;
            v[2] = dp;
            v[3] = dp;
            v[4] = b + 1;
            v[5] = (unsigned long long)(ld * 1024.0);
            v[6] = (unsigned long long)(ld * ld * 1024.0);
        }
        const int32_t u0 = __shfl_sync(0xffffffffu, u, 0);
        if (__all_sync(0xffffffffu, ok && u == u0)) {
            for (int o = 16; o; o >>= 1) {
                v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
                v[1] += __shfl_xor_sync(0xffffffffu, v[1], o);
                v[2] += __shfl_xor_sync(0xffffffffu, v[2], o);
                v[3] = max(v[3], __shfl_xor_sync(0xffffffffu, v[3], o));
                v[4] = max(v[4], __shfl_xor_sync(0xffffffffu, v[4], o));
                v[5] += __shfl_xor_sync(0xffffffffu, v[5], o);
                v[6] += __shfl_xor_sync(0xffffffffu, v[6], o);
            }
            if (lane != 0) continue;
        } else if (!ok) {
            continue;
        }
        unsigned long long* o = out + (uint64_t)u * kRawStats;
        atomicAdd(&o[0], v[0]);
        atomicAdd(&o[1], v[1]);
        atomicAdd(&o[2], v[2]);
        atomicMax(&o[3], v[3]);
        atomicMax(&o[4], v[4]);
        atomicAdd(&o[6], v[5]);
        atomicAdd(&o[7], v[6]);
    }
}

// In-edge statistics: a warp per vertex c streams its prefix N+(c); every
// pivot b there has c as an in-neighbour and gains dplus[c] (the bound on
// c's scan).  Lanes hitting the same unit are merged with __match_any_sync;
// with kSmem (up to kScanStatsSmemUnits units) the per-unit sums gather in a
// shared-memory histogram first, because almost every row starts with hub
// ids and global atomics on the first units would serialise.
constexpr uint32_t kScanStatsSmemUnits = 4096;

template <bool kSmem>
__global__ void k_unit_scan_stats(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj,
                                  const uint32_t* __restrict__ dplus, const int32_t* __restrict__ unit_of,
                                  uint64_t n, uint32_t U, unsigned long long* __restrict__ out) {
    extern __shared__ unsigned long long hist[];  // kSmem: 2 U counters (scan bound, long prefixes)
    if (kSmem) {
        for (uint32_t i = threadIdx.x; i < 2 * U; i += blockDim.x) hist[i] = 0;
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t c = warp; c < n; c += nwarps) {
        const uint32_t dc = dplus[c];
        if (dc == 0) continue;
        const int32_t* row = adj + off[c];
        for (uint32_t k0 = 0; k0 < dc; k0 += 32) {
            const uint32_t k = k0 + lane;
            const bool ok = k < dc;
            const int32_t u = ok ? unit_of[row[k]] : -1;
            const unsigned peers = __match_any_sync(0xffffffffu, u);
            if (ok && lane == __ffs(peers) - 1) {
                const unsigned long long cntp = (unsigned long long)__popc(peers);
                if (kSmem) {
                    atomicAdd(&hist[2 * u], cntp * dc);
                    if (dc >= 32) atomicAdd(&hist[2 * u + 1], cntp);
                } else {
                    atomicAdd(&out[(uint64_t)u * kRawStats + 5], cntp * dc);
                    if (dc >= 32) atomicAdd(&out[(uint64_t)u * kRawStats + 8], cntp);
                }
            }
        }
    }
    if (kSmem) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < U; i += blockDim.x) {
            if (hist[2 * i]) atomicAdd(&out[(uint64_t)i * kRawStats + 5], hist[2 * i]);
            if (hist[2 * i + 1]) atomicAdd(&out[(uint64_t)i * kRawStats + 8], hist[2 * i + 1]);
        }
    }
}

// First CSR entry of pivot b's in-neighbours at or above c_min (0: of all).
__device__ __forceinline__ uint64_t first_in_neighbour(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj,
                                                       const uint32_t* __restrict__ dplus, int32_t b, int32_t c_min) {
    const uint64_t in0 = off[b] + dplus[b];
    return c_min > b ? in0 + lower_bound_i32(adj + in0, (uint32_t)(off[b + 1] - in0), c_min) : in0;
}

// One launch's list of work items.
struct ItemList {
    Item* items;
    uint32_t* count;  // zeroed before
    uint32_t cap;     // room of items: an upper bound of the count
    uint32_t chunk;   // in-neighbours per item
    int32_t c_min;    // in-neighbours below this are not taken
};

// Work items of all launches of a count: pivot b gives its list (list_of[its
// unit], -1: none) ceil(din / chunk) items, each a run of <= chunk of its
// in-neighbours; pivots without a set or without in-neighbours give none.
//
// A warp takes a block of 32 kRows consecutive pivots.  The lists are in pivot
// order wherever a block has pivots of one list only: kItemsCount writes the
// blocks' items, k_item_offsets adds them up per list, kItemsOrdered fills them
// in.  (In the order of an atomic per block the bitmap kernels of RMAT-20 took
// 873 instead of 798 us: sets of neighbouring pivots are scanned by rows that
// L2 still holds.)  Blocks with several lists, and all blocks of small graphs
// (kItemsAny, a single pass), take an atomic per list instead.  A count, a scan
// and a fill per launch cost 20 us for each of them.
enum ItemPass { kItemsCount, kItemsOrdered, kItemsAny };
struct __align__(16) ItemBlock {
    uint32_t n;     // items
    uint32_t at;    // the block's first place in its list
    int32_t list;   // -1: none, -2: several
    int32_t pad;
};
// The items of a block of hubs (100 K for RMAT-24's first one) are written by
// kRows warps, a row of pivots each.
constexpr uint32_t kItemsSplit = 256;

template <int kRows, int kPass>
__global__ void k_items(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj,
                        const uint32_t* __restrict__ dplus, const int32_t* __restrict__ unit_of,
                        const int16_t* __restrict__ list_of, const ItemList* __restrict__ lists, uint64_t n,
                        ItemBlock* __restrict__ blocks) {
    const int lane = threadIdx.x & 31;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const int part = blockIdx.y;  // kItemsOrdered: 0 .. kRows - 1
    for (uint64_t blk = warp; blk * 32 * kRows < n; blk += nwarps) {
        const bool split = kPass == kItemsOrdered && blocks[blk].n > kItemsSplit;
        if (part && !split) continue;
        const uint64_t b0 = blk * 32 * kRows;
        uint64_t in0[kRows];
        uint32_t din[kRows], c[kRows];
        int32_t l[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const uint64_t b = min(b0 + 32 * i + lane, n - 1);
            const uint32_t dp = dplus[b];
            in0[i] = off[b] + dp;
            din[i] = (uint32_t)(off[b + 1] - in0[i]);
            l[i] = unit_of[b];
            if (dp == 0 || b0 + 32 * i + lane >= n) din[i] = 0;
        }
        uint32_t sum = 0;
        int32_t mine = -1;  // the lane's list, -2: more than one
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            c[i] = 0;
            l[i] = din[i] ? list_of[l[i]] : -1;
            if (l[i] < 0) continue;
            const int32_t c_min = lists[l[i]].c_min;
            if (c_min) {
                const uint64_t b = b0 + 32 * i + lane;
                in0[i] = first_in_neighbour(off, adj, dplus, (int32_t)b, c_min);
                din[i] = (uint32_t)(off[b + 1] - in0[i]);
            }
            const uint32_t chunk = lists[l[i]].chunk;
            c[i] = (din[i] + chunk - 1) / chunk;
            if (!c[i]) continue;
            sum += c[i];
            mine = mine == -1 || mine == l[i] ? l[i] : -2;
        }
        const unsigned have = __ballot_sync(0xffffffffu, sum != 0);
        const int32_t l0 = have ? __shfl_sync(0xffffffffu, mine, __ffs(have) - 1) : -1;
        const bool one = __all_sync(0xffffffffu, sum == 0 || mine == l0) && l0 >= 0;
        if (kPass == kItemsCount) {
            for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            if (lane == 0) blocks[blk] = ItemBlock{one ? sum : 0u, 0u, have ? (one ? l0 : -2) : -1, 0};
            continue;
        }
        if (!have) continue;
        // the lists of the block one after the other
        for (unsigned left = have; left;) {
            int32_t cur = 0x7fffffff;  // the smallest list not done yet
#pragma unroll
            for (int i = 0; i < kRows; ++i)
                if (c[i]) cur = min(cur, l[i]);
            cur = __reduce_min_sync(0xffffffffu, cur);
            uint32_t own = 0;
#pragma unroll
            for (int i = 0; i < kRows; ++i)
                if (c[i] && l[i] == cur) own += c[i];
            uint32_t end = own;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, end, o);
                if (lane >= o) end += x;
            }
            const ItemList L = lists[cur];
            uint32_t at = 0;
            if (lane == 31) at = kPass == kItemsOrdered && one ? blocks[blk].at : atomicAdd(L.count, end);
            at = __shfl_sync(0xffffffffu, at, 31) + end - own;
            bool more = false;
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const int32_t b = (int32_t)(b0 + 32 * i + lane);
                const uint32_t ci = l[i] == cur ? c[i] : 0u;
                const bool here = !split || i == part;
                if (here && ci && ci <= 8)
                    for (uint32_t j = 0; j < ci && at + j < L.cap; ++j)
                        L.items[at + j] = Item{in0[i] + (uint64_t)j * L.chunk, b, min(L.chunk, din[i] - j * L.chunk)};
                // a hub's items are written by the warp together
                for (unsigned hubs = __ballot_sync(0xffffffffu, here && ci > 8); hubs; hubs &= hubs - 1) {
                    const int src = __ffs(hubs) - 1;
                    const uint32_t cs = __shfl_sync(0xffffffffu, ci, src), as = __shfl_sync(0xffffffffu, at, src);
                    const uint32_t ds = __shfl_sync(0xffffffffu, din[i], src);
                    const uint64_t is = __shfl_sync(0xffffffffu, in0[i], src);
                    for (uint32_t j = lane; j < cs && as + j < L.cap; j += 32)
                        L.items[as + j] = Item{is + (uint64_t)j * L.chunk, b - lane + src, min(L.chunk, ds - j * L.chunk)};
                }
                at += ci;
                if (ci) c[i] = 0;
                more |= c[i] != 0;
            }
            left = __ballot_sync(0xffffffffu, more);
        }
    }
}

// Finds the blocks' first places in their list and writes the list's length
// (of the ordered blocks).  A CTA per list, a run of blocks per warp.
__global__ void __launch_bounds__(1024) k_item_offsets(ItemBlock* __restrict__ blocks, uint32_t nblocks,
                                                       const ItemList* __restrict__ lists) {
    __shared__ uint32_t s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l = blockIdx.x;
    const uint32_t per = ((nblocks + 1023) / 1024) * 32, k0 = min(nblocks, warp * per), k1 = min(nblocks, k0 + per);
    uint32_t own = 0;
#pragma unroll 8
    for (uint32_t k = k0 + lane; k < k1; k += 32) {
        const ItemBlock B = blocks[k];
        if (B.list == l) own += B.n;
    }
    own = __reduce_add_sync(0xffffffffu, own);
    if (lane == 0) s_warp[warp] = own;
    __syncthreads();
    uint32_t at = 0, total = 0;
    for (int w = 0; w < 32; ++w) {
        if (w < warp) at += s_warp[w];
        total += s_warp[w];
    }
    if (threadIdx.x == 0) *lists[l].count = total;
    if (own == 0) return;
    for (uint32_t kk = k0; kk < k1; kk += 32) {
        const uint32_t k = kk + lane;
        const bool mine = k < k1 && blocks[k].list == l;
        const uint32_t c = mine ? blocks[k].n : 0u;
        uint32_t end = c;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += x;
        }
        if (mine) blocks[k].at = at + end - c;
        at += __shfl_sync(0xffffffffu, end, 31);
    }
}

// The items of bitmap lists by where their in-neighbours' rows lie in the
// oriented copy: kBins parts of equal size, in list order (about) within a part.
// In pivot order every pivot sweeps the rows of all its in-neighbours, and on a
// graph whose rows L2 does not hold the scans of the hub units wait on DRAM
// (4.5-5.9 TB/s in RMAT-24's).  An item builds its pivot's set either way.
constexpr int kBins = 64;
__device__ __forceinline__ int bin_of(const Item& I, const int32_t* __restrict__ adj, const uint32_t* __restrict__ ooff,
                                      uint64_t vecs) {
    return min((int)((uint64_t)ooff[adj[I.in0]] * kBins / vecs), kBins - 1);
}

__global__ void k_bin_count(const Item* __restrict__ items, const uint32_t* __restrict__ nitems, uint32_t cap,
                            const int32_t* __restrict__ adj, const uint32_t* __restrict__ ooff, uint64_t vecs,
                            uint32_t* __restrict__ bins) {
    __shared__ uint32_t h[kBins];
    if (threadIdx.x < kBins) h[threadIdx.x] = 0;
    __syncthreads();
    const uint32_t n = min(*nitems, cap);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(&h[bin_of(items[i], adj, ooff, vecs)], 1u);
    __syncthreads();
    if (threadIdx.x < kBins && h[threadIdx.x]) atomicAdd(&bins[threadIdx.x], h[threadIdx.x]);
}

// bins: the counts, then kBins zeroed words (items placed so far).
__global__ void k_bin_scatter(const Item* __restrict__ items, const uint32_t* __restrict__ nitems, uint32_t cap,
                              const int32_t* __restrict__ adj, const uint32_t* __restrict__ ooff, uint64_t vecs,
                              uint32_t* __restrict__ bins, Item* __restrict__ out) {
    __shared__ uint32_t base[kBins], h[kBins], at[kBins];
    if (threadIdx.x == 0) {
        uint32_t sum = 0;
        for (int k = 0; k < kBins; ++k) {
            base[k] = sum;
            sum += bins[k];
        }
    }
    const uint32_t n = min(*nitems, cap);
    for (uint64_t tile = blockIdx.x * (uint64_t)blockDim.x; tile < n; tile += (uint64_t)gridDim.x * blockDim.x) {
        if (threadIdx.x < kBins) h[threadIdx.x] = 0;
        __syncthreads();
        const uint64_t i = tile + threadIdx.x;
        Item I{};
        int k = 0;
        uint32_t rank = 0;
        if (i < n) {
            I = items[i];
            k = bin_of(I, adj, ooff, vecs);
            rank = atomicAdd(&h[k], 1u);
        }
        __syncthreads();
        if (threadIdx.x < kBins)
            at[threadIdx.x] = base[threadIdx.x] +
                              (h[threadIdx.x] ? atomicAdd(&bins[kBins + threadIdx.x], h[threadIdx.x]) : 0u);
        __syncthreads();
        if (i < n) out[at[k] + rank] = I;
    }
}

// H[b - lo][a >> 5] |= bit(a) for a in N+(b), one warp per pivot.
__global__ void k_matrix_rows(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj,
                              const uint32_t* __restrict__ dplus, int32_t lo, int32_t hi, uint32_t hstride,
                              uint32_t* __restrict__ H) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t b = lo + warp; b < hi; b += nwarps) {
        const int32_t* row = adj + off[b];
        uint32_t* h = H + (uint64_t)(b - lo) * hstride;
        for (uint32_t k = lane; k < dplus[b]; k += 32) {
            const int32_t a = row[k];
            atomicOr(&h[a >> 5], 1u << (a & 31));
        }
    }
}

// Word form of a block whose last pivot b sits at position jl: ceil(b/128)
// 16-byte words per row against ceil(jl/32) probe rounds.
__device__ __forceinline__ bool matrix_words_win(int32_t b, uint32_t jl) {
    const uint32_t nv = ((((uint32_t)b + 31) >> 5) + 3) >> 2;
    return ((nv + 31) >> 5) < ((jl + 31) >> 5);
}

// The pairs (b, c) of one in-neighbour c: S = N(c) & [0, min(hi, c)), pivots
// at positions [j0, k).  Pivots are taken U consecutive positions at a time,
// so each step of the warp has U independent row loads in flight per lane and
// shares one load of S (or of its bitmap) between them (RMAT-24 count with
// U = 4: 27.7 ms, 8: 27.1; RMAT-22: 4.51 and 4.50):
//  - probe form: lanes read S[i] for i below the block's last position and
//    test bit S[i] of each pivot's row (i < j of that pivot);
//  - word form: lanes AND 16-byte words of each row with the warp's
//    shared-memory bitmap of S and count bits.  A row b has bits only below
//    b, so words past a pivot's own length read zeros.
// The form is chosen per block by the rounds each needs; the bitmap is built
// only when some block uses it.
__device__ __forceinline__ unsigned long long matrix_block_pairs(const int32_t* S, uint32_t j0, uint32_t k,
                                                                 int32_t lo, uint32_t hstride,
                                                                 const uint32_t* __restrict__ H, uint32_t* Sb,
                                                                 int lane) {
    constexpr int U = kMatrixBlock;
    unsigned long long cnt = 0;
    bool want = false;
    for (uint32_t jb = j0 + (uint32_t)lane * U; jb < k; jb += 32u * U) {
        const uint32_t jl = min(jb + (uint32_t)U, k) - 1;
        want |= matrix_words_win(S[jl], jl);
    }
    const bool words = __any_sync(0xffffffffu, want);
    if (words) {
        for (uint32_t i = lane; i < k; i += 32) {
            const int32_t a = S[i];
            atomicOr(&Sb[a >> 5], 1u << (a & 31));
        }
        __syncwarp();
    }
    const uint4* Sb4 = reinterpret_cast<const uint4*>(Sb);
    for (uint32_t jb = j0; jb < k; jb += U) {
        const uint32_t ju = min((uint32_t)U, k - jb), jl = jb + ju - 1;
        const int32_t bl = S[jl];
        const uint32_t* h[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int32_t b = (uint32_t)u < ju ? S[jb + u] : bl;
            h[u] = H + (uint64_t)(b - lo) * hstride;
        }
        if (words && matrix_words_win(bl, jl)) {
            const uint32_t nv = ((((uint32_t)bl + 31) >> 5) + 3) >> 2;
            for (uint32_t x = lane; x < nv; x += 32) {
                const uint4 sv = Sb4[x];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if ((uint32_t)u < ju) {
                        const uint4 v = __ldg(reinterpret_cast<const uint4*>(h[u]) + x);
                        cnt += __popc(v.x & sv.x) + __popc(v.y & sv.y) + __popc(v.z & sv.z) + __popc(v.w & sv.w);
                    }
                }
            }
        } else {
            for (uint32_t i = lane; i < jl; i += 32) {
                const int32_t a = S[i];
                const uint32_t w = (uint32_t)a >> 5, bit = (uint32_t)a & 31;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if ((uint32_t)u < ju && i < jb + (uint32_t)u) cnt += (__ldg(h[u] + w) >> bit) & 1u;
            }
        }
    }
    if (words) {
        __syncwarp();
        for (uint32_t i = lane; i < k; i += 32) Sb[S[i] >> 5] = 0;
        __syncwarp();
    }
    return cnt;
}

// Pivot positions [klo, khi) of in-neighbour c in its row (N(c) is sorted,
// and min(hi, c) <= c keeps the search inside N+(c)).
__device__ __forceinline__ void matrix_span(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj,
                                            const uint32_t* __restrict__ dplus, int32_t lo, int32_t hi, uint64_t c,
                                            uint64_t* r, uint32_t* klo, uint32_t* khi) {
    *r = off[c];
    const int32_t lim = (int64_t)c < (int64_t)hi ? (int32_t)c : hi;
    *khi = lower_bound_i32(adj + *r, dplus[c], lim);
    *klo = lower_bound_i32(adj + *r, *khi, lo);
}

// The in-neighbours c in (lo, c1), taken one per warp: they are the hubs, with
// long spans S_c (c1: kMatrixFrom).
__global__ void __launch_bounds__(kMatrixWarps * 32) k_tc_matrix(const uint64_t* __restrict__ off,
                                                               const int32_t* __restrict__ adj,
                                                               const uint32_t* __restrict__ dplus, int32_t lo,
                                                               int32_t hi, uint64_t c1, uint32_t hstride,
                                                               const uint32_t* __restrict__ H,
                                                               unsigned long long* __restrict__ next,
                                                               unsigned long long* __restrict__ total,
                                                               unsigned long long* __restrict__ unit_cost,
                                                               int32_t unit) {
    extern __shared__ uint4 msm4[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t* Sb = reinterpret_cast<uint32_t*>(msm4) + (size_t)w * hstride;  // warp-private bitmap of S_c
    for (uint32_t i = lane; i < hstride; i += 32) Sb[i] = 0;
    __syncwarp();
    const long long t0 = unit_cost ? clock64() : 0;
    unsigned long long cnt = 0;
    for (;;) {
        unsigned long long q = 0;
        if (lane == 0) q = atomicAdd(next, 1ull);
        const uint64_t c = __shfl_sync(0xffffffffu, q, 0) + (uint64_t)lo + 1;
        if (c >= c1) break;
        uint64_t r = 0;
        uint32_t klo = 0, khi = 0;
        if (lane == 0) matrix_span(off, adj, dplus, lo, hi, c, &r, &klo, &khi);
        r = __shfl_sync(0xffffffffu, r, 0);
        klo = __shfl_sync(0xffffffffu, klo, 0);
        khi = __shfl_sync(0xffffffffu, khi, 0);
        if (khi > klo) cnt += matrix_block_pairs(adj + r, klo, khi, lo, hstride, H, Sb, lane);
    }
    if (unit_cost) {
        __syncwarp();
        if (lane == 0) atomicAdd(&unit_cost[unit], (unsigned long long)(clock64() - t0));
    }
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0 && cnt) atomicAdd(total, cnt);
}

// A matrix unit's in-neighbours from this id on run through the bitmap kernel:
// their spans are short, and the probes of a short span into rows of L2 are
// slower than a scan against a bitmap in shared memory.  RMAT-24 / RMAT-22
// counts in ms with the line at 2^13: 33.6 / 5.15, 2^14: 31.6 / 4.85,
// 2^15: 30.0 / 4.55, 2^16: 27.1 / 4.50, 2^17: 27.1 / 4.57, 2^18: 27.3 / 4.66,
// 2^19: 28.0 / 4.80.
constexpr int32_t kMatrixFrom = 1 << 16;

constexpr uint32_t kBitmapCapBits = 1u << 20;  // 128 KB of shared memory

static bool bitmap_feasible(const float* f) { return f[4] <= (float)kBitmapCapBits; }
// The in-neighbour-major form needs the unit's pivots to be the id range
// [lo, hi) (contiguous partitions; tc_assign checks that) with hi <= 2^16,
// and its resident rows to fit L2 (126 MB on B200): rows that spill re-read
// DRAM on every probe, which is what the form exists to avoid (RMAT-24's
// fourth hub unit, 128 MB of rows, cost 4 ms more than the bitmap kernel).
constexpr double kMatrixRowsCap = 100.0 * (1 << 20);
static bool matrix_feasible(const float* f) {
    const double words = (double)((((uint64_t)f[4] + 31) / 32 + 3) & ~(uint64_t)3);
    return f[4] <= (float)kMatrixMaxId && (double)f[0] * words * 4.0 <= kMatrixRowsCap;
}

// Plain autotuned heuristic.  Thresholds come from heuristic_params(), which
// the autotuner (pc_selector_autotune) may replace.
int heuristic_choice(const float* f, const HeuristicParams& hp) {
    const double npiv = f[0], ein = f[1], sdp = f[2], mdp = f[3];
    if (ein <= 0 || sdp <= 0) return -1;
    const double scan = f[5] / std::max(1.0, ein);
    const double inpp = ein / std::max(1.0, npiv);
    if (matrix_feasible(f) && inpp >= hp.min_in_per_pivot_cta && scan >= hp.matrix_scan) return PC_VARIANT_MATRIX;
    if (bitmap_feasible(f) && inpp >= hp.min_in_per_pivot_cta) {
        if (scan >= hp.warp_scan) return PC_VARIANT_BITMAP_WARP;
        if (scan >= hp.group_scan) return PC_VARIANT_BITMAP_GROUP8;
        return PC_VARIANT_BITMAP_LANE;
    }
    if (mdp <= kHashCap) return PC_VARIANT_HASH_WARP;
    if (bitmap_feasible(f)) return PC_VARIANT_BITMAP_GROUP8;
    return PC_VARIANT_MERGE_LANE;
}

bool variant_feasible(int v, const float* f) {
    switch (v) {
        case PC_VARIANT_BITMAP_WARP:
        case PC_VARIANT_BITMAP_GROUP8:
        case PC_VARIANT_BITMAP_LANE: return bitmap_feasible(f);
        case PC_VARIANT_MATRIX: return matrix_feasible(f);
        default: return v >= 0 && v < PC_NUM_VARIANTS;
    }
}

static bool is_bitmap(int v) {
    return v == PC_VARIANT_BITMAP_WARP || v == PC_VARIANT_BITMAP_GROUP8 || v == PC_VARIANT_BITMAP_LANE;
}

// Bitmap sets per CTA: K warps share one set, 16 / K sets per CTA.  The
// smallest K whose CTAs (sets and the per-vertex mode's hub histogram) stay
// below a third of an SM's shared memory, or a half, or all of it: the scans
// wait on L2, so resident warps come before sets of fewer warps.
struct BitmapShape {
    int K;
    uint32_t words;
    size_t smem;
    int ctas_per_sm;
};

static void fill_shape(BitmapShape* sh, int mode, int kind) {
    sh->smem = (size_t)(16 / sh->K) * bitmap_set_words(sh->words, mode, kind) * 4 +
               (mode == kCountVertex ? (size_t)kHubHist * 4 : 0);
    // 1 KB a CTA is the system's
    sh->ctas_per_sm = (int)std::min<size_t>(4, 227 * 1024 / (sh->smem + 1280));
}

static BitmapShape bitmap_shape(uint32_t words, int mode) {
    BitmapShape sh{};
    sh.words = words;
    for (int per_sm = 3; per_sm >= 1; --per_sm)
        for (sh.K = 1; sh.K <= 16; sh.K *= 2) {
            fill_shape(&sh, mode, kPlainSet);
            if (sh.ctas_per_sm >= per_sm) return sh;
        }
    sh.K = 16;
    fill_shape(&sh, mode, kPlainSet);
    return sh;
}

// Mixed sets of K warps with `lo` low ids.  kSplitLo: the bitmap units, two
// warps a set: 7.2 KB sets, so three CTAs and 48 warps stay on an SM (RMAT-24's
// units of ids 65-196 K: 7.23 ms; 2^16 low ids in 10 KB sets of four warps,
// whose barriers cost more, 8.27 ms).  kLightLo: the light pivots of the hash
// variant, a set per warp of 4 KB: 2^13 exact low ids keep most look-ups away
// (RMAT-24 4.16 ms, RMAT-16 0.16 ms in all, against 4.25 and 0.19 ms with lo = 0;
// ER-20, whose ids spread evenly, 0.98 against 0.88 ms).
constexpr uint32_t kSplitLo = 1u << 15, kLightLo = 1u << 13;
constexpr uint32_t kSplitFrom = 1u << 16;  // bitmap units with pivots past this id have mixed sets
static BitmapShape mixed_shape(int mode, int K, uint32_t lo) {
    BitmapShape sh{};
    sh.K = K;
    sh.words = lo / 32 + kFilterWords;
    fill_shape(&sh, mode, kMixedSet);
    return sh;
}

// Arguments of one bitmap-kernel launch.
struct BitmapLaunch {
    unsigned grid;
    size_t smem;
    cudaStream_t s;
    OrientedView oriented;    // ids null: scans of the CSR
    CsrView csr;
    const int32_t* adj;
    const Item* items;
    const uint32_t* nitems;
    uint32_t cap;
    uint32_t* next;
    unsigned long long* total;
    uint32_t words;
    unsigned long long* cost;
    const int32_t* unit_of;
    unsigned long long* tri;  // per-vertex triangle counts (LCC), or null
    uint32_t* ecnt;           // per-edge counts at the oriented slots (Jaccard), or null
};

template <int K, int G, int V, int kMode, int kKind, class Rows>
static pc_status launch_bitmap_rows(const Rows& R, const BitmapLaunch& L) {
    auto* kernel = k_tc_bitmap<K, G, V, kMode, kKind, Rows>;
    PC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem));
    kernel<<<L.grid, kCtaThreads, L.smem, L.s>>>(R, L.adj, L.items, L.nitems, L.cap, L.next, L.total, L.words, L.cost,
                                                 L.unit_of, L.tri, L.ecnt);
    return PC_OK;
}

// G: lanes per in-neighbour on the copy (the CSR is scanned with 4); light: one vector a step.
template <int K, int kMode, int kKind>
static pc_status launch_bitmap_kmode(int G, bool light, const BitmapLaunch& L) {
    constexpr int V = kMode == kCountEdge ? 1 : 2;
    if (light) {
        if constexpr (K == 1 && kKind == kMixedSet) {
            if (!L.oriented.ids) return launch_bitmap_rows<1, 4, 1, kMode, kMixedSet>(L.csr, L);
            return launch_bitmap_rows<1, 4, 1, kMode, kMixedSet>(L.oriented, L);
        }
        return fail(PC_ERR_UNSUPPORTED, "light pivot sets: unexpected launch shape");
    }
    if constexpr (!(K == 1 && kKind == kMixedSet)) {
        if (!L.oriented.ids) return launch_bitmap_rows<K, 4, V, kMode, kKind>(L.csr, L);
        if (G == 32) return launch_bitmap_rows<K, 32, 1, kMode, kKind>(L.oriented, L);
        if (G == 8) return launch_bitmap_rows<K, 4, V, kMode, kKind>(L.oriented, L);
        return launch_bitmap_rows<K, 1, 1, kMode, kKind>(L.oriented, L);
    }
    return fail(PC_ERR_UNSUPPORTED, "mixed pivot sets: unexpected launch shape");
}

template <int K>
static pc_status launch_bitmap_k(int G, const BitmapLaunch& L) {
    if (L.tri) return launch_bitmap_kmode<K, kCountVertex, kPlainSet>(G, false, L);
    if (L.ecnt) return launch_bitmap_kmode<K, kCountEdge, kPlainSet>(G, false, L);
    return launch_bitmap_kmode<K, kCountOnly, kPlainSet>(G, false, L);
}

static pc_status launch_bitmap(int K, int G, int kind, const BitmapLaunch& L) {
    if (kind == kMixedSet) {  // fixed-size sets (mixed_shape): light pivots with a set per warp
        if (K == 1 && L.ecnt) return launch_bitmap_kmode<1, kCountEdge, kMixedSet>(G, true, L);
        if (K == 1 && L.tri) return launch_bitmap_kmode<1, kCountVertex, kMixedSet>(G, true, L);
        if (K == 1) return launch_bitmap_kmode<1, kCountOnly, kMixedSet>(G, true, L);
        if (L.ecnt || K != 2) return fail(PC_ERR_UNSUPPORTED, "mixed pivot sets: unexpected launch shape");
        if (L.tri) return launch_bitmap_kmode<2, kCountVertex, kMixedSet>(G, false, L);
        return launch_bitmap_kmode<2, kCountOnly, kMixedSet>(G, false, L);
    }
    switch (K) {
        case 1: return launch_bitmap_k<1>(G, L);
        case 2: return launch_bitmap_k<2>(G, L);
        case 4: return launch_bitmap_k<4>(G, L);
        case 8: return launch_bitmap_k<8>(G, L);
        default: return launch_bitmap_k<16>(G, L);
    }
}

}  // namespace tc

using namespace tc;

static pc_status tc_features(pc_pgraph* pg) {
    PC_TRY(ensure_dplus(pg));
    build_units(pg, &pg->unit_lo, &pg->unit_hi);
    const size_t U = pg->unit_lo.size();
    const uint64_t n = pg->g->n;
    pg->part_features.assign(U * kNumFeatures, 0.f);
    if (U == 0) return PC_OK;
    PC_TRY(pg->unit_of.ensure(std::max<uint64_t>(n, 1) * 4, "unit of vertex"));
    PC_TRY(scratch_reserve(pg, U * 16 + U * kRawStats * 8));
    int64_t* d_lo = nullptr;
    int64_t* d_hi = nullptr;
    PC_TRY(upload(pg, pg->unit_lo.data(), U, &d_lo));
    PC_TRY(upload(pg, pg->unit_hi.data(), U, &d_hi));
    unsigned long long* d_raw = pg->scratch.take<unsigned long long>(U * kRawStats);
    cudaStream_t s = pg->g->stream;
    PC_CUDA(cudaMemsetAsync(d_raw, 0, U * kRawStats * 8, s));
    const int32_t* plist = pg->contiguous ? nullptr : pg->new2old.as<int32_t>();
    int32_t* unit_of = pg->unit_of.as<int32_t>();
    const int sms = sm_count(pg->g->device);
    k_unit_of<<<(unsigned)U, 256, 0, s>>>(plist, d_lo, d_hi, unit_of);
    PC_LAUNCHED();
    k_unit_pivot_stats<<<sms * 8, 256, 0, s>>>(pg->off, pg->dplus.as<uint32_t>(), unit_of, n, d_raw);
    PC_LAUNCHED();
    if (U <= kScanStatsSmemUnits) {
        const size_t smem = 2 * U * sizeof(unsigned long long);
        PC_CUDA(cudaFuncSetAttribute(k_unit_scan_stats<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_unit_scan_stats<true><<<sms * 2, 1024, smem, s>>>(pg->off, pg->adj, pg->dplus.as<uint32_t>(), unit_of, n,
                                                           (uint32_t)U, d_raw);
    } else {
        k_unit_scan_stats<false><<<sms * 16, 256, 0, s>>>(pg->off, pg->adj, pg->dplus.as<uint32_t>(), unit_of, n,
                                                           (uint32_t)U, d_raw);
    }
    PC_LAUNCHED();
    std::vector<unsigned long long> raw(U * kRawStats);
    PC_CUDA(cudaMemcpyAsync(raw.data(), d_raw, raw.size() * 8, cudaMemcpyDeviceToHost, s));
    PC_TRY(sync(pg));
    for (size_t u = 0; u < U; ++u) raw_to_features(&raw[u * kRawStats], &pg->part_features[u * kNumFeatures]);
    return PC_OK;
}

pc_status tc_ensure_features(pc_pgraph* pg) {
    if (pg->features_ready) return PC_OK;
    PC_TRY(tc_features(pg));
    pg->features_ready = true;
    return PC_OK;
}

// Item lists are binned where L2 (126 MB) does not hold the oriented copy: counts
// of RMAT-24 27.1 -> 25.0 ms, RMAT-22 (0.27 GB) 4.50 -> 4.40, but RMAT-20 (65 MB)
// 0.99 -> 1.02, where the rows stay in L2 in any order.
constexpr uint64_t kBinFrom = 126ull << 20;

// One launch: a variant and its bitmap shape (words rounded up to a power
// of two).
struct LaunchGroup {
    int v = -1;
    uint32_t words = 0;
    bool split = false;  // bitmap variants: mixed sets
    std::vector<int64_t> ranges;
    uint64_t npos = 0, item_bound = 0;
    double ein = 0;
    size_t units = 0;
    std::vector<int32_t> unit_ids;  // matrix groups: one launch per unit (ranges not merged)
    int32_t c_min = 0;              // in-neighbours below this are not taken
    std::vector<LaunchGroup> tails; // matrix groups: the in-neighbours from kMatrixFrom on, per bitmap shape
    // launches of item lists (finish_group)
    BitmapShape shape{};
    uint32_t chunk = 0;
    bool binned = false;            // items in order of their in-neighbours' rows
    int list = -1;                  // index among the count's lists
    ItemList dev{};
};

// Words per resident pivot bitmap row of a matrix unit with ids below hi:
// ceil(hi / 32) rounded up to 16 bytes, so rows can be read as uint4.
static uint32_t matrix_stride(int64_t hi) { return (uint32_t)((((hi + 31) / 32) + 3) & ~(int64_t)3); }

// Bytes of the resident pivot bitmap rows of a matrix unit [lo, hi).
static uint64_t matrix_bytes(int64_t lo, int64_t hi) { return (uint64_t)(hi - lo) * matrix_stride(hi) * 4; }

// Bitmap units whose pivot ids pass kSplitFrom run with mixed sets in
// the count and per-vertex modes, unless PC_BITMAP_SPLIT=0 is in the
// environment (read once; a switch for measurements).
static bool bitmap_split_enabled() {
    static const bool on = [] {
        const char* e = getenv("PC_BITMAP_SPLIT");
        return !(e && atoi(e) == 0);
    }();
    return on;
}

static pc_status launch_matrix(pc_pgraph* pg, int64_t lo, int64_t hi, uint32_t hstride, const uint32_t* H,
                               unsigned long long* d_next, unsigned long long* d_total, unsigned long long* d_cost,
                               int32_t unit, int sms, cudaStream_t s) {
    const size_t smem = (size_t)kMatrixWarps * hstride * 4;
    PC_CUDA(cudaFuncSetAttribute(k_tc_matrix, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    PC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tc_matrix, kMatrixWarps * 32, smem));
    const uint64_t c1 = std::min<uint64_t>(pg->g->n, (uint64_t)kMatrixFrom);
    k_tc_matrix<<<(unsigned)(sms * std::max(1, per_sm)), kMatrixWarps * 32, smem, s>>>(
        pg->off, pg->adj, pg->dplus.as<uint32_t>(), (int32_t)lo, (int32_t)hi, c1, hstride, H, d_next, d_total, d_cost, unit);
    PC_LAUNCHED();
    return PC_OK;
}

// The in-neighbour-major form over one unit (ids [lo, hi)), all asynchronous:
// rows H built from N+(b), then the walk over the in-neighbours.
static pc_status run_matrix_unit(pc_pgraph* pg, int64_t lo, int64_t hi, int32_t unit, uint32_t* H,
                                 unsigned long long* d_next, unsigned long long* d_total, unsigned long long* d_cost,
                                 uint64_t* launches) {
    cudaStream_t s = pg->g->stream;
    const int sms = sm_count(pg->g->device);
    const uint32_t hstride = matrix_stride(hi);
    PC_CUDA(cudaMemsetAsync(H, 0, matrix_bytes(lo, hi), s));
    PC_CUDA(cudaMemsetAsync(d_next, 0, 16, s));
    k_matrix_rows<<<sms * 8, 256, 0, s>>>(pg->off, pg->adj, pg->dplus.as<uint32_t>(), (int32_t)lo, (int32_t)hi, hstride,
                                          H);
    PC_LAUNCHED();
    PC_TRY(launch_matrix(pg, lo, hi, hstride, H, d_next, d_total, d_cost, unit, sms, s));
    *launches += 2;
    return PC_OK;
}

// Shape and item size of a launch.  An item is up to 256 in-neighbours per warp
// of its set, less where that would leave sets without one: RMAT-10's 11 K
// in-edges in runs of 256 kept one warp busy for 30 us, in runs of 32 for 13.
// Items never exceed min(pivots, in-edges) + in-edges / chunk; the float
// in-edge feature is widened by 256 per unit for its rounding.
static void finish_group(LaunchGroup* gr, int mode, int sms) {
    const uint64_t ein = (uint64_t)gr->ein + 256 * gr->units;
    uint64_t per_set = 0, sets = 0, most = 0;
    if (is_bitmap(gr->v) || gr->v == PC_VARIANT_HASH_WARP) {
        if (gr->v == PC_VARIANT_HASH_WARP) gr->shape = mixed_shape(mode, 1, mode == kCountEdge ? 0u : kLightLo);
        else gr->shape = gr->split ? mixed_shape(mode, 2, kSplitLo) : bitmap_shape(gr->words, mode);
        per_set = 32u * (uint32_t)gr->shape.K;
        sets = (uint64_t)sms * gr->shape.ctas_per_sm * (16 / gr->shape.K);
        most = 256u * (uint32_t)gr->shape.K;
    } else {
        per_set = 32;
        sets = (uint64_t)sms * 8 * kWarpCtaWarps;
        most = (uint64_t)kChunkWarp;
    }
    const uint64_t want = ceil_div(ceil_div(ein, 2 * sets), per_set) * per_set;
    gr->chunk = (uint32_t)std::min(most, std::max(per_set, want));
    gr->item_bound = std::min<uint64_t>(gr->npos, ein) + ein / gr->chunk + 1;
}

static pc_status run_items(pc_pgraph* pg, const LaunchGroup& gr, unsigned long long* d_total, uint64_t* launches,
                           unsigned long long* d_cost, unsigned long long* d_tri, uint32_t* d_ecnt);

// Launches one group (all asynchronous).
static pc_status run_group(pc_pgraph* pg, const LaunchGroup& gr, unsigned long long* d_total, uint64_t* launches,
                           unsigned long long* d_cost, unsigned long long* d_tri, uint32_t* d_ecnt) {
    if (gr.v == PC_VARIANT_MATRIX) {
        uint64_t hb = 0;
        for (size_t i = 0; i < gr.unit_ids.size(); ++i) hb = std::max(hb, matrix_bytes(gr.ranges[2 * i], gr.ranges[2 * i + 1]));
        uint32_t* H = pg->scratch.take<uint32_t>(hb / 4);
        unsigned long long* d_next = pg->scratch.take<unsigned long long>(2);
        if (!H || !d_next) return fail(PC_ERR_OOM, "scratch arena too small (internal sizing error)");
        for (size_t i = 0; i < gr.unit_ids.size(); ++i)
            PC_TRY(run_matrix_unit(pg, gr.ranges[2 * i], gr.ranges[2 * i + 1], gr.unit_ids[i], H, d_next, d_total,
                                   d_cost, launches));
        for (const LaunchGroup& t : gr.tails) PC_TRY(run_items(pg, t, d_total, launches, d_cost, d_tri, d_ecnt));
        return PC_OK;
    }
    return run_items(pg, gr, d_total, launches, d_cost, d_tri, d_ecnt);
}


// The groups whose work is a list of items (built by k_items).
static pc_status run_items(pc_pgraph* pg, const LaunchGroup& gr, unsigned long long* d_total, uint64_t* launches,
                           unsigned long long* d_cost, unsigned long long* d_tri, uint32_t* d_ecnt) {
    const int32_t* unit_of = pg->unit_of.as<int32_t>();
    cudaStream_t s = pg->g->stream;
    const int v = gr.v;
    const uint32_t* dp = pg->dplus.as<uint32_t>();
    const int sms = sm_count(pg->g->device);
    if (gr.npos == 0) return PC_OK;
    const BitmapShape& sh = gr.shape;
    const bool light = v == PC_VARIANT_HASH_WARP;
    const Item* d_items = gr.dev.items;
    const uint32_t* d_nitems = gr.dev.count;
    uint32_t* d_next = gr.dev.count + 1;
    if (is_bitmap(v) || light) {  // run by k_tc_bitmap
        BitmapLaunch L;
        L.smem = sh.smem;
        L.grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)sms * sh.ctas_per_sm, gr.item_bound));
        L.s = s;
        L.oriented = OrientedView{pg->ooff.as<uint32_t>(), pg->oids.as<int4>()};
        L.csr = CsrView{pg->off, pg->adj, dp, 0};
        L.adj = pg->adj;
        L.items = d_items;
        L.nitems = d_nitems;
        L.cap = gr.dev.cap;
        L.next = d_next;
        L.total = d_total;
        L.words = sh.words;
        L.cost = d_cost;
        L.unit_of = unit_of;
        L.tri = d_tri;
        L.ecnt = d_ecnt;
        const int Gsel = v == PC_VARIANT_BITMAP_WARP ? 32 : (v == PC_VARIANT_BITMAP_GROUP8 ? 8 : 1);
        PC_TRY(launch_bitmap(sh.K, Gsel, light || gr.split ? kMixedSet : kPlainSet, L));
    } else {
        const unsigned grid = (unsigned)std::max<uint64_t>(
            1, std::min<uint64_t>((uint64_t)sms * 8, ceil_div(gr.item_bound, kWarpCtaWarps)));
        const unsigned bs = kWarpCtaWarps * 32;
        const uint32_t* ooff = pg->oids.p ? pg->ooff.as<uint32_t>() : nullptr;
        auto launch = [&](auto* kernel) {
            kernel<<<grid, bs, 0, s>>>(pg->off, pg->adj, dp, ooff, d_items, d_nitems, gr.dev.cap, d_next, d_total, d_cost, unit_of,
                                       d_tri, d_ecnt);
        };
        if (v == PC_VARIANT_MERGE_LANE) {
            if (d_ecnt) launch(k_tc_warp<kModeMerge, false, true>);
            else if (d_tri) launch(k_tc_warp<kModeMerge, true>);
            else launch(k_tc_warp<kModeMerge>);
        } else {
            if (d_ecnt) launch(k_tc_warp<kModeGallop, false, true>);
            else if (d_tri) launch(k_tc_warp<kModeGallop, true>);
            else launch(k_tc_warp<kModeGallop>);
        }
    }
    PC_LAUNCHED();
    *launches += 1;
    return PC_OK;
}

// Executes an assignment (one launch group per variant and bitmap shape
// used) and returns the count; the only host synchronisation is the final
// 8-byte read.  With unit_ms (profiling runs) the kernels also charge their
// warp-cycles to the units, every group is timed by its own events, and each
// unit gets its group's time in proportion to its cycles: the unit's cost
// inside a full run, where it shares the GPU with the other units.
static pc_status tc_execute(pc_pgraph* pg, const std::vector<int8_t>& assign, uint64_t* count, pc_tc_stats* stats,
                            std::vector<double>* unit_ms = nullptr, unsigned long long* d_tri = nullptr,
                            uint32_t* d_ecnt = nullptr) {
    cudaStream_t s = pg->g->stream;
    const std::vector<int64_t>& lo = pg->unit_lo;
    const std::vector<int64_t>& hi = pg->unit_hi;
    const std::vector<float>& feat = pg->part_features;
    const size_t U = lo.size();
    // Bitmap units are grouped by their bitmap size rounded up to a power of
    // two, so the hub units (small ids) get small sets and more CTAs per SM;
    // in the count and per-vertex modes, units with pivot ids past
    // kSplitFrom share one group of fixed-size mixed sets (class kClasses).
    constexpr int kClasses = 16;
    const bool split_ok = bitmap_split_enabled() && !d_ecnt;
    std::vector<LaunchGroup> groups(PC_NUM_VARIANTS * (kClasses + 1));
    std::vector<int> group_of(U, -1);
    for (size_t u = 0; u < U; ++u) {
        const int v = assign[u];
        if (v < 0) continue;
        const uint32_t mid = (uint32_t)feat[u * kNumFeatures + 4];
        auto bitmap_class = [&]() {
            const uint32_t w = std::max<uint32_t>(1, (mid + 31) / 32);
            int c = 0;
            while ((1u << c) < w && c < kClasses - 1) ++c;
            return split_ok && mid > kSplitFrom ? kClasses : c;
        };
        auto add_unit = [&](LaunchGroup& gr, bool merge) {
            if (merge && !gr.ranges.empty() && gr.ranges.back() == lo[u]) {
                gr.ranges.back() = hi[u];
            } else {
                gr.ranges.push_back(lo[u]);
                gr.ranges.push_back(hi[u]);
            }
            gr.npos += (uint64_t)(hi[u] - lo[u]);
            gr.ein += feat[u * kNumFeatures + 1];
            gr.units += 1;
        };
        const int c = is_bitmap(v) ? bitmap_class() : 0;
        LaunchGroup& gr = groups[v * (kClasses + 1) + c];
        group_of[u] = v * (kClasses + 1) + c;
        gr.v = v;
        gr.split = c == kClasses;
        gr.words = gr.split ? 0 : 1u << c;
        add_unit(gr, v != PC_VARIANT_MATRIX);
        if (v != PC_VARIANT_MATRIX) continue;
        gr.unit_ids.push_back((int32_t)u);
        if ((uint64_t)kMatrixFrom >= pg->g->n) continue;
        const int tc = bitmap_class();
        LaunchGroup* tail = nullptr;
        for (LaunchGroup& t : gr.tails)
            if (t.words == 1u << tc) tail = &t;
        if (!tail) {
            gr.tails.emplace_back();
            tail = &gr.tails.back();
            tail->v = PC_VARIANT_BITMAP_GROUP8;
            tail->words = 1u << tc;
            tail->c_min = kMatrixFrom;
        }
        add_unit(*tail, true);
    }
    const int mode = d_tri ? kCountVertex : (d_ecnt ? kCountEdge : kCountOnly);
    const int sms = sm_count(pg->g->device);
    std::vector<LaunchGroup*> listed;  // the groups with an item list
    size_t need = 4096, need_binned = 0;
    // lists put in order of their in-neighbours' rows
    const uint64_t n = pg->g->n;
    const bool bin = n >= (1u << 17) && pg->oids.p && pg->ovecs * 16 > kBinFrom;
    auto add_list = [&](LaunchGroup& gr) {
        finish_group(&gr, mode, sms);
        gr.list = (int)listed.size();
        listed.push_back(&gr);
        gr.binned = bin && is_bitmap(gr.v);
        const size_t room = gr.item_bound * sizeof(Item) + 256 + kBins * 8;
        need += room;
        if (gr.binned) need_binned += room;
    };
    for (LaunchGroup& gr : groups) {
        if (gr.ranges.empty()) continue;
        if (gr.v == PC_VARIANT_MATRIX) {
            uint64_t hb = 0;
            for (size_t i = 0; i < gr.unit_ids.size(); ++i)
                hb = std::max(hb, matrix_bytes(gr.ranges[2 * i], gr.ranges[2 * i + 1]));
            need += hb + 2 * 256;
            for (LaunchGroup& t : gr.tails) add_list(t);
            continue;
        }
        add_list(gr);
    }
    // the list of every unit (a matrix unit's is its tail's)
    std::vector<int16_t> list_of(std::max<size_t>(U, 1), -1);
    for (const LaunchGroup* gr : listed)
        for (size_t i = 0; i < gr->ranges.size(); i += 2) {
            const size_t u0 = std::lower_bound(lo.begin(), lo.end(), gr->ranges[i]) - lo.begin();
            for (size_t u = u0; u < U && lo[u] < gr->ranges[i + 1]; ++u) list_of[u] = (int16_t)gr->list;
        }
    // ordered lists from 2^17 vertices on; below, three launches cost more
    // (RMAT-16 0.15 ms with them, 0.11 without)
    const uint64_t item_blocks = n >= (1u << 17) ? ceil_div(n, 256) : 0;
    need += U * 2 + listed.size() * (sizeof(ItemList) + 8) + item_blocks * sizeof(ItemBlock) + 1024;
    if (unit_ms) need += U * 8 + 256;
    pc_status reserved = scratch_reserve(pg, need + need_binned);
    if (reserved == PC_ERR_OOM && need_binned) {  // the lists in pivot order need half the room
        for (LaunchGroup* gr : listed) gr->binned = false;
        clear_error();
        reserved = scratch_reserve(pg, need);
    }
    PC_TRY(reserved);
    // the total, then a count and a taken-items counter per list
    unsigned long long* d_total = pg->scratch.take<unsigned long long>(1 + listed.size());
    int16_t* d_list_of = nullptr;
    ItemList* d_lists = nullptr;
    ItemBlock* d_blocks = item_blocks ? pg->scratch.take<ItemBlock>(item_blocks) : nullptr;
    if (item_blocks && !d_blocks) return fail(PC_ERR_OOM, "scratch arena too small (internal sizing error)");
    std::vector<ItemList> lists(listed.size());
    for (size_t i = 0; i < listed.size(); ++i) {
        ItemList& L = listed[i]->dev;
        L.items = pg->scratch.take<Item>(listed[i]->item_bound);
        if (!L.items) return fail(PC_ERR_OOM, "scratch arena too small (internal sizing error)");
        L.count = reinterpret_cast<uint32_t*>(d_total + 1 + i);
        L.cap = (uint32_t)listed[i]->item_bound;
        L.chunk = listed[i]->chunk;
        L.c_min = listed[i]->c_min;
        lists[i] = L;
    }
    unsigned long long* d_cost = unit_ms ? pg->scratch.take<unsigned long long>(std::max<size_t>(U, 1)) : nullptr;
    std::vector<cudaEvent_t> gev;
    auto drop_events = [&]() {
        for (cudaEvent_t e : gev) cudaEventDestroy(e);
        gev.clear();
    };
    if (unit_ms) {
        gev.resize(2 * groups.size(), nullptr);
        for (cudaEvent_t& e : gev)
            if (cudaEventCreate(&e) != cudaSuccess) {
                drop_events();
                return fail(PC_ERR_CUDA, "event creation failed");
            }
        PC_CUDA(cudaMemsetAsync(d_cost, 0, std::max<size_t>(U, 1) * 8, s));
    }
    uint64_t launches = 0;
    if (stats) PC_CUDA(cudaEventRecord(pg->ev0, s));
    PC_CUDA(cudaMemsetAsync(d_total, 0, 8 * (1 + listed.size()), s));
    if (!listed.empty()) {
        // one copy: the lists, then the units' list numbers
        std::vector<char> tables(lists.size() * sizeof(ItemList) + U * 2);
        memcpy(tables.data(), lists.data(), lists.size() * sizeof(ItemList));
        memcpy(tables.data() + lists.size() * sizeof(ItemList), list_of.data(), U * 2);
        char* d_tables = nullptr;
        PC_TRY(upload(pg, tables.data(), tables.size(), &d_tables));
        d_lists = reinterpret_cast<ItemList*>(d_tables);
        d_list_of = reinterpret_cast<int16_t*>(d_tables + lists.size() * sizeof(ItemList));
        auto launch = [&](auto* kernel, int rows, unsigned parts) {  // rows: pivots per lane
            const dim3 grid((unsigned)std::min<uint64_t>((uint64_t)sms * 16, ceil_div(n, 128 * rows)), parts);
            kernel<<<grid, 128, 0, s>>>(
                pg->off, pg->adj, pg->dplus.as<uint32_t>(), pg->unit_of.as<int32_t>(), d_list_of, d_lists, n, d_blocks);
        };
        if (item_blocks) {
            launch(k_items<8, kItemsCount>, 8, 1);
            PC_LAUNCHED();
            k_item_offsets<<<(unsigned)listed.size(), 1024, 0, s>>>(d_blocks, (uint32_t)item_blocks, d_lists);
            PC_LAUNCHED();
            launch(k_items<8, kItemsOrdered>, 8, 8);
            launches += 2;
        } else {
            launch(k_items<1, kItemsAny>, 1, 1);
        }
        PC_LAUNCHED();
        ++launches;
        for (LaunchGroup* gr : listed) {
            if (!gr->binned) continue;
            Item* sorted = pg->scratch.take<Item>(gr->item_bound);
            uint32_t* bins = pg->scratch.take<uint32_t>(2 * kBins);
            if (!sorted || !bins) return fail(PC_ERR_OOM, "scratch arena too small (internal sizing error)");
            PC_CUDA(cudaMemsetAsync(bins, 0, 2 * kBins * 4, s));
            const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)sms * 8, ceil_div(gr->item_bound, 256));
            const uint32_t* ooff = pg->ooff.as<uint32_t>();
            k_bin_count<<<grid, 256, 0, s>>>(gr->dev.items, gr->dev.count, gr->dev.cap, pg->adj, ooff, pg->ovecs, bins);
            PC_LAUNCHED();
            k_bin_scatter<<<grid, 256, 0, s>>>(gr->dev.items, gr->dev.count, gr->dev.cap, pg->adj, ooff, pg->ovecs, bins,
                                               sorted);
            PC_LAUNCHED();
            gr->dev.items = sorted;
            launches += 2;
        }
    }
    for (size_t gi = 0; gi < groups.size(); ++gi) {
        const LaunchGroup& gr = groups[gi];
        if (gr.ranges.empty()) continue;
        if (unit_ms) PC_CUDA(cudaEventRecord(gev[2 * gi], s));
        PC_TRY(run_group(pg, gr, d_total, &launches, d_cost, d_tri, d_ecnt));
        if (unit_ms) PC_CUDA(cudaEventRecord(gev[2 * gi + 1], s));
    }
    if (stats) PC_CUDA(cudaEventRecord(pg->ev1, s));
    unsigned long long h = 0;
    PC_CUDA(cudaMemcpyAsync(&h, d_total, 8, cudaMemcpyDeviceToHost, s));
    std::vector<unsigned long long> cyc(unit_ms ? U : 0);
    if (unit_ms && U) PC_CUDA(cudaMemcpyAsync(cyc.data(), d_cost, U * 8, cudaMemcpyDeviceToHost, s));
    const pc_status st = sync(pg);
    if (st != PC_OK) {
        drop_events();
        return st;
    }
    *count = h;
    if (unit_ms) {
        unit_ms->assign(U, 0.0);
        std::vector<double> gsum(groups.size(), 0.0), gms(groups.size(), 0.0);
        for (size_t u = 0; u < U; ++u)
            if (group_of[u] >= 0) gsum[group_of[u]] += (double)cyc[u];
        for (size_t gi = 0; gi < groups.size(); ++gi) {
            if (groups[gi].ranges.empty()) continue;
            float ms = 0.f;
            cudaEventElapsedTime(&ms, gev[2 * gi], gev[2 * gi + 1]);
            gms[gi] = ms;
        }
        for (size_t u = 0; u < U; ++u) {
            const int gi = group_of[u];
            if (gi >= 0 && gsum[gi] > 0) (*unit_ms)[u] = gms[gi] * (double)cyc[u] / gsum[gi];
        }
        drop_events();
    }
    if (stats) {
        memset(stats, 0, sizeof(*stats));
        stats->partitions = pg->P;
        for (size_t u = 0; u < U; ++u)
            if (assign[u] >= 0) stats->variant_hist[assign[u]]++;
        float ms = 0.f;
        PC_CUDA(cudaEventElapsedTime(&ms, pg->ev0, pg->ev1));
        stats->kernel_ms = ms;
        stats->launches = launches;
        double w = 0;
        for (size_t u = 0; u < U; ++u) w += feat_raw_scan(&feat[u * kNumFeatures]);
        stats->scan_bound = (uint64_t)w;
    }
    return PC_OK;
}

// Chooses a variant per unit.
pc_status tc_assign(pc_pgraph* pg, int32_t variant, const std::vector<float>& feat, size_t U,
                    std::vector<int8_t>* assign, int* selector_used) {
    assign->assign(U, -1);
    if (variant >= 0) {
        if (variant >= PC_NUM_VARIANTS) return fail(PC_ERR_INVALID_INPUT, "unknown TC variant");
        if (variant == PC_VARIANT_MATRIX && !pg->contiguous)
            return fail(PC_ERR_UNSUPPORTED, "forced matrix variant: the partitions are not contiguous id ranges");
        for (size_t u = 0; u < U; ++u) {
            const float* f = &feat[u * kNumFeatures];
            if (f[1] <= 0 || f[2] <= 0) continue;
            if (!variant_feasible(variant, f))
                return fail(PC_ERR_UNSUPPORTED, variant == PC_VARIANT_MATRIX
                                                    ? "forced matrix variant: a pivot id is 2^16 or above, or a unit's rows exceed 100 MB"
                                                    : "forced bitmap variant: a pivot id exceeds the shared-memory "
                                                      "bitmap capacity");
            (*assign)[u] = (int8_t)variant;
        }
        *selector_used = 0;
        return PC_OK;
    }
    if (variant != PC_VARIANT_AUTO && variant != PC_VARIANT_HEURISTIC)
        return fail(PC_ERR_INVALID_INPUT, "unknown TC variant");
    const bool learned = (variant == PC_VARIANT_AUTO) && selector_ready(pg->g->device);
    const uint64_t key = selector_version() * 4 + (learned ? 1 : 0);
    if (pg->plan_key == key && pg->plan_assign.size() == U) {
        *assign = pg->plan_assign;
        *selector_used = learned ? 2 : 1;
        return PC_OK;
    }
    HeuristicParams hp = heuristic_params();
    // the matrix form needs units that are id ranges
    if (!pg->contiguous) hp.matrix_scan = INFINITY;
    if (learned) PC_TRY(selector_choose_batch(feat, U, assign));
    for (size_t u = 0; u < U; ++u) {
        const float* f = &feat[u * kNumFeatures];
        if (f[1] <= 0 || f[2] <= 0) { (*assign)[u] = -1; continue; }
        int v = learned ? (*assign)[u] : heuristic_choice(f, hp);
        if (v < 0 || !variant_feasible(v, f) || (v == PC_VARIANT_MATRIX && !pg->contiguous))
            v = heuristic_choice(f, hp);
        (*assign)[u] = (int8_t)v;
    }
    pg->plan_key = key;
    pg->plan_assign = *assign;
    *selector_used = learned ? 2 : 1;
    return PC_OK;
}

static pc_status tc_count_run(pc_pgraph* pg, int32_t variant, uint64_t* count, pc_tc_stats* stats) {
    PC_TRY(ensure_oriented(pg));
    PC_TRY(tc_ensure_features(pg));
    const size_t U = pg->unit_lo.size();
    if (U == 0 || pg->g->m == 0) {
        *count = 0;
        if (stats) memset(stats, 0, sizeof(*stats));
        return PC_OK;
    }
    std::vector<int8_t> assign;
    int sel = 0;
    PC_TRY(tc_assign(pg, variant, pg->part_features, U, &assign, &sel));
    PC_TRY(tc_execute(pg, assign, count, stats));
    if (stats) stats->selector = sel;
    return PC_OK;
}

pc_status tc_count(pc_pgraph* pg, int32_t variant, uint64_t* count, pc_tc_stats* stats) {
    return with_room(pg, [&] { return tc_count_run(pg, variant, count, stats); });
}

// Per-vertex triangle counts (each triangle adds 1 to each of its three
// vertices) into d_tri (n zeroed counters, outside the scratch arena) under
// the plan of `variant`; the matrix form has no per-vertex mode, so its units
// run with the 32-lane bitmap kernel.  Returns the triangle count.
pc_status tc_vertex_triangles(pc_pgraph* pg, int32_t variant, unsigned long long* d_tri, uint64_t* count) {
    PC_TRY(ensure_oriented(pg));
    PC_TRY(tc_ensure_features(pg));
    const size_t U = pg->unit_lo.size();
    *count = 0;
    if (U == 0 || pg->g->m == 0) return PC_OK;
    std::vector<int8_t> assign;
    int sel = 0;
    PC_TRY(tc_assign(pg, variant, pg->part_features, U, &assign, &sel));
    for (size_t u = 0; u < U; ++u) {
        if (assign[u] != PC_VARIANT_MATRIX) continue;
        const float* f = &pg->part_features[u * kNumFeatures];
        assign[u] = (int8_t)(bitmap_feasible(f) ? PC_VARIANT_BITMAP_WARP : PC_VARIANT_HASH_WARP);
    }
    return tc_execute(pg, assign, count, nullptr, nullptr, d_tri);
}

// Counters tc_edge_triangles needs.  Builds the oriented copy or not, which
// decides where the slots are, so tc_edge_triangles itself leaves that alone.
pc_status tc_edge_slots(pc_pgraph* pg, uint64_t* slots) {
    PC_TRY(ensure_oriented(pg));
    PC_TRY(tc_ensure_features(pg));
    *slots = pg->oids.p ? 4 * pg->ovecs : pg->g->m;
    return PC_OK;
}

// Per-edge triangle counts at the oriented slots (the slot of edge {x, y},
// y < x, is the position of y in row x of the oriented copy, see slot_base)
// into d_ecnt (tc_edge_slots zeroed counters, outside the scratch arena),
// under the plan of `variant`; matrix units run with the 32-lane bitmap
// kernel.  Returns the triangle count.
pc_status tc_edge_triangles(pc_pgraph* pg, int32_t variant, uint32_t* d_ecnt, uint64_t* count) {
    PC_TRY(tc_ensure_features(pg));
    const size_t U = pg->unit_lo.size();
    *count = 0;
    if (U == 0 || pg->g->m == 0) return PC_OK;
    std::vector<int8_t> assign;
    int sel = 0;
    PC_TRY(tc_assign(pg, variant, pg->part_features, U, &assign, &sel));
    for (size_t u = 0; u < U; ++u) {
        if (assign[u] != PC_VARIANT_MATRIX) continue;
        const float* f = &pg->part_features[u * kNumFeatures];
        assign[u] = (int8_t)(bitmap_feasible(f) ? PC_VARIANT_BITMAP_WARP : PC_VARIANT_HASH_WARP);
    }
    return tc_execute(pg, assign, count, nullptr, nullptr, nullptr, d_ecnt);
}

// Runs one variant on every unit it can take (all units with work; bitmap
// variants only where the ids fit) in one profiled call; returns the per-unit
// cost inside that full run, -1 where the variant cannot run, and the count
// over the units it ran.
static pc_status tc_profile_variant_run(pc_pgraph* pg, int variant, std::vector<double>* unit_ms, uint64_t* count) {
    PC_TRY(ensure_oriented(pg));
    PC_TRY(tc_ensure_features(pg));
    const size_t U = pg->unit_lo.size();
    std::vector<int8_t> assign(U, -1);
    const bool ok = variant != PC_VARIANT_MATRIX || pg->contiguous;
    for (size_t u = 0; u < U; ++u) {
        const float* f = &pg->part_features[u * kNumFeatures];
        if (ok && f[1] > 0 && f[2] > 0 && variant_feasible(variant, f)) assign[u] = (int8_t)variant;
    }
    PC_TRY(tc_execute(pg, assign, count, nullptr, unit_ms));
    for (size_t u = 0; u < U; ++u)
        if (assign[u] < 0) (*unit_ms)[u] = -1.0;
    return PC_OK;
}

pc_status tc_profile_variant(pc_pgraph* pg, int variant, std::vector<double>* unit_ms, uint64_t* count) {
    return with_room(pg, [&] { return tc_profile_variant_run(pg, variant, unit_ms, count); });
}

// Times one variant on one unit alone (selector training data).
static pc_status tc_time_unit_run(pc_pgraph* pg, size_t unit, int variant, double* ms, uint64_t* count) {
    PC_TRY(ensure_oriented(pg));
    PC_TRY(tc_ensure_features(pg));
    const size_t U = pg->unit_lo.size();
    if (unit >= U) return fail(PC_ERR_INVALID_INPUT, "unit index out of range");
    std::vector<int8_t> assign(U, -1);
    assign[unit] = (int8_t)variant;
    pc_tc_stats st;
    PC_TRY(tc_execute(pg, assign, count, &st));
    *ms = st.kernel_ms;
    return PC_OK;
}

pc_status tc_time_unit(pc_pgraph* pg, size_t unit, int variant, double* ms, uint64_t* count) {
    return with_room(pg, [&] { return tc_time_unit_run(pg, unit, variant, ms, count); });
}

}  // namespace pc

using namespace pc;

extern "C" {

pc_status pc_tc_ex(pc_pgraph* pg, int32_t method, int32_t variant, uint64_t* count, pc_tc_stats* stats) {
    clear_error();
    if (!pg || !count) return fail(PC_ERR_INVALID_INPUT, "null argument");
    if (method != PC_METHOD_MERGE && method != PC_METHOD_GALLOPING) return fail(PC_ERR_INVALID_INPUT, "unknown method");
    PC_TRY(use_device(pg->g));
    uint64_t t = 0;
    PC_TRY(tc_count(pg, variant, &t, stats));
    // The galloping form sums |N(u) & N(v)| over every ordered edge (u, v),
    // which counts each triangle 6 times (src/Graph.cpp:1326-1344).
    *count = method == PC_METHOD_MERGE ? t : 6 * t;
    return PC_OK;
}

pc_status pc_tc(pc_pgraph* pg, int32_t method, uint64_t* count) {
    return pc_tc_ex(pg, method, PC_VARIANT_AUTO, count, nullptr);
}

}  // extern "C"
