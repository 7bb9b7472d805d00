// Many independent graphs in one launch: triangle counts per graph, LCC per
// vertex and BFS levels per vertex (from each graph's first vertex).
//
// The graphs are packed in one CSR arena with arena-wide vertex ids; graph g
// owns vertices [voff[g], voff[g+1]) and no edge joins two graphs, so the
// arena is one block-diagonal graph.  A single persistent kernel first takes
// the BFS items (a graph each, largest first, one CTA) and then the triangle
// items (a pivot and a run of its in-neighbours, one warp) from global
// counters: no CTA ever waits for another, so the launch needs no grid-wide
// synchronisation, and a large graph's triangles are spread over the whole
// GPU.  One enumeration serves both the counts and the coefficients.  The
// launch sequence (clears, the kernel, the coefficients' division, the result
// copies) is captured once into a CUDA graph and replayed by later calls; the
// schedule (threads per CTA, CTAs per SM, BFS order) comes from
// pc_batch_autotune.
//
// Measured against one CTA per (graph, task), whose launch lasted as long as
// its largest graph: 96 graphs of scales 8..12 (4.2 M entries) 7.0 -> 0.26 ms
// on the device, 4096 graphs of scales 10..16 (2.4 G entries) 1261 -> 134 ms.
// Bound by instruction issue in the scans (scan_in_neighbours), and for a few
// small graphs by the latency of one CTA's BFS levels.
#include <algorithm>
#include <climits>
#include <cstring>
#include <numeric>
#include <string>
#include <vector>

#include "pc_internal.cuh"
#include "tc_kernels.cuh"

struct pc_batch {
    pc_graph* g = nullptr;  // the arena (validated by pc_graph_create)
    uint32_t G = 0;
    std::vector<uint64_t> voff;
    std::vector<uint64_t> gm;  // directed edges per graph
    pc::DevBuf d_voff, dplus, ooff, oids, titems, tri, dist, q0, q1, tc, items, counter;
    uint64_t ovecs = 0;
    uint32_t ntri = 0;  // triangle items
    uint64_t* h_tc = nullptr;  // pinned staging
    double* h_lcc = nullptr;
    int32_t* h_bfs = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    uint64_t exec_key = ~0ull;
    int threads = 512, ctas_per_sm = 2, order = 0;
    uint32_t nitems = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

namespace pc {
namespace bt {

constexpr int kMaxWarps = 16;
constexpr int32_t kLowIds = 1 << 13;  // graph-local ids with exact bits (mixed sets, a set per warp)
constexpr uint32_t kBits = kLowIds / 32 + tc::kFilterWords;
constexpr int32_t kHubs = 512;        // graph-local ids whose triangles each warp gathers in shared memory (LCC)
constexpr uint32_t kSetWords = tc::bitmap_set_words(kBits, tc::kCountOnly, tc::kMixedSet);
constexpr uint32_t kWarpWords(bool lcc) { return kSetWords + (lcc ? (uint32_t)kHubs : 0u); }
constexpr uint32_t kHeavyRow = 256;   // BFS: longer frontier rows are expanded by the whole CTA
constexpr uint32_t kHeavyList = 256;  // ... up to so many a level
constexpr uint32_t kItemRun = 256;  // in-neighbours per triangle item

// base[v]: the first vertex of v's graph (v's graph-local id is v - base[v]).
// Needed for the preparation only, in the memory of the BFS queues.
__global__ void k_graph_of(const uint64_t* __restrict__ voff, int32_t* __restrict__ graph_of,
                           int32_t* __restrict__ base) {
    const uint64_t v0 = voff[blockIdx.x], v1 = voff[blockIdx.x + 1];
    for (uint64_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
        graph_of[v] = (int32_t)blockIdx.x;
        base[v] = (int32_t)v0;
    }
}

__global__ void k_prepare(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj,
                          const uint64_t* __restrict__ voff, const int32_t* __restrict__ graph_of, uint64_t n,
                          uint32_t* __restrict__ dplus, uint32_t* __restrict__ bad) {
    const uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (u >= n) return;
    const uint64_t b = off[u], e = off[u + 1];
    if (e > b) {
        const int32_t g = graph_of[u];
        if ((uint64_t)adj[b] < voff[g] || (uint64_t)adj[e - 1] >= voff[g + 1]) atomicOr(bad, 1u);
    }
    uint64_t lo = b, hi = e;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (adj[mid] < (int32_t)u) lo = mid + 1; else hi = mid;
    }
    dplus[u] = (uint32_t)(lo - b);
}

// Triangle items: every pivot with a set and in-neighbours gives a run of
// items of <= kItemRun in-neighbours, appended in any order (items null: counted
// only).  The in-neighbours are found from the pivot, so that a sparse arena's
// items take no more room than the counts and coefficients leave.
struct TriItem {
    int32_t b;     // pivot
    int32_t g;     // its graph
    uint32_t run;  // in-neighbours from run * kItemRun on
};

__global__ void k_triangle_items(const uint64_t* __restrict__ off, const uint32_t* __restrict__ dplus,
                                 const int32_t* __restrict__ graph_of, uint64_t n, TriItem* __restrict__ items,
                                 uint32_t* __restrict__ nitems) {
    const uint64_t b = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (b >= n || dplus[b] == 0) return;
    const uint64_t din = off[b + 1] - off[b] - dplus[b];
    const uint32_t c = (uint32_t)((din + kItemRun - 1) / kItemRun);
    if (!c) return;
    const uint32_t s = atomicAdd(nitems, c);
    if (items)
        for (uint32_t j = 0; j < c; ++j) items[s + j] = TriItem{(int32_t)b, graph_of[b], j};
}

struct Args {
    const uint64_t* off;
    const int32_t* adj;
    const uint64_t* voff;
    const uint32_t* dplus;
    tc::OrientedView oriented;  // rows in graph-local ids; ids null: the CSR's
    const TriItem* titems;
    uint32_t ntri;
    const int32_t* bfs_order;   // graphs to search, in this order
    uint32_t nbfs;
    uint32_t* counter;          // [0] next BFS item, [1] next triangle item
    unsigned long long* tc;     // per graph, or null
    unsigned long long* tri;    // per vertex (LCC), or null
    int32_t* dist;
    int32_t* q0;
    int32_t* q1;
};

// The triangle items, one warp each, with a mixed pivot set of graph-local ids
// (exact bits below kLowIds, which holds the hubs of every graph of the
// batch).  kMode kCountVertex also counts each vertex's triangles; a warp
// gathers those of a graph's first kHubs vertices, where nearly every hit
// lands, in shared memory and adds them up when it comes to another graph
// (one global atomic per hit: 1.05 ms for 96 graphs of 4.2 M entries).
template <int kMode, class Rows>
__device__ __forceinline__ void warp_triangles(const Args& A, Rows R, uint32_t* bm) {
    const int lane = threadIdx.x & 31;
    int32_t* ht = reinterpret_cast<int32_t*>(bm + kBits);
    for (uint32_t i = lane; i < kBits; i += 32) bm[i] = 0;
    for (uint32_t i = lane; i < (uint32_t)tc::kHashSlots; i += 32) ht[i] = -1;
    uint32_t* hist = bm + kSetWords;
    int32_t hist_base = -1;
    if (kMode == tc::kCountVertex)
        for (int i = lane; i < kHubs; i += 32) hist[i] = 0;
    __syncwarp();
    auto flush = [&]() {
        if (kMode != tc::kCountVertex || hist_base < 0) return;
        __syncwarp();
        for (int i = lane; i < kHubs; i += 32) {
            const uint32_t h = hist[i];
            if (h) {
                atomicAdd(&A.tri[hist_base + i], (unsigned long long)h);
                hist[i] = 0;
            }
        }
        __syncwarp();
    };
    for (;;) {
        uint32_t it = 0;
        if (lane == 0) it = atomicAdd(&A.counter[1], 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= A.ntri) break;
        const TriItem I = A.titems[it];
        const int32_t base = (int32_t)A.voff[I.g], b = I.b - base;
        const uint64_t in0 = A.off[I.b] + A.dplus[I.b] + (uint64_t)I.run * kItemRun;
        const uint32_t nin = (uint32_t)min((uint64_t)kItemRun, A.off[I.b + 1] - in0);
        if constexpr (Rows::kCsr) R.base = base;
        if (base != hist_base) {
            flush();
            hist_base = base;
        }
        const typename Rows::Row row = R.row(I.b);
        tc::SetView S;
        S.bm = bm;
        S.lo = kLowIds;
        S.ht = ht;
        S.hpos = nullptr;
        R.sorted(row, &S);
        S.ovf = S.np > (uint32_t)tc::kHashCap && __ldg(S.nb + (S.np - tc::kHashCap - 1)) - S.base >= kLowIds;
        bool high = false;
        for (uint32_t k = lane; k < row.n; k += 32) {
            const int4 v = R.vector(row, k);
            const int32_t e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int32_t a = e[t];
                if (a == INT32_MAX) continue;  // padding
                const uint32_t x = S.place<tc::kMixedSet>(a);
                atomicOr(&bm[x >> 5], 0x80000000u >> (x & 31));
                if (!S.ovf && a >= kLowIds) {
                    high = true;
                    uint32_t hs = tc::hash_slot(a);
                    while (atomicCAS(&ht[hs], -1, a) != -1) hs = (hs + 1) & (tc::kHashSlots - 1);
                }
            }
        }
        __syncwarp();
        tc::HitSink sink;
        sink.tri = A.tri;
        sink.tri_low = A.tri + base;
        sink.hist = hist;
        sink.hist_ids = kHubs;
        sink.by_slot = sink.used = nullptr;
        sink.ecnt = sink.by_rank = nullptr;
        sink.ranks = tc::SetRanks{nullptr, nullptr};
        unsigned long long hits = 0;
        for (uint32_t k = 0; k < nin; k += 32) {
            const int nb = min(32, (int)(nin - k));
            const int32_t c = lane < nb ? A.adj[in0 + k + lane] : 0;
            hits += tc::scan_in_neighbours<4, 1, kMode, tc::kMixedSet>(R, c, nb, b, S, lane, sink);
        }
        for (int o = 16; o; o >>= 1) hits += __shfl_xor_sync(0xffffffffu, hits, o);
        if (lane == 0 && hits) {
            if (A.tc) atomicAdd(&A.tc[I.g], hits);
            if (kMode == tc::kCountVertex) atomicAdd(&A.tri[I.b], hits);
        }
        for (uint32_t k = lane; k < row.n; k += 32) {
            const int4 v = R.vector(row, k);
            bm[S.place<tc::kMixedSet>(v.x) >> 5] = 0;
            bm[S.place<tc::kMixedSet>(v.y) >> 5] = 0;
            bm[S.place<tc::kMixedSet>(v.z) >> 5] = 0;
            bm[S.place<tc::kMixedSet>(v.w) >> 5] = 0;
        }
        if (__any_sync(0xffffffffu, high))
            for (uint32_t i = lane; i < (uint32_t)tc::kHashSlots; i += 32) ht[i] = -1;
        __syncwarp();
    }
    flush();
}

// LCC from per-vertex triangle counts, as in intersect.cu
// (src/Graph.cpp:833-838), each in the place of its count.
__global__ void k_batch_lcc(const uint64_t* __restrict__ off, uint64_t n, unsigned long long* __restrict__ tri) {
    const uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (u >= n) return;
    const uint64_t du = off[u + 1] - off[u];
    tri[u] = __double_as_longlong(du < 1 ? 0.0 : (double)(2 * tri[u]) / (double)(du * (du - 1)));
}

// Level-synchronous BFS of one graph by one CTA, direction-optimising (Beamer,
// Asanovic, Patterson, SC'12).  Top-down: a warp per frontier vertex; rows of
// more than kHeavyRow entries are set aside and expanded by all warps, so
// that a hub does not hold the level up with one dependent load after
// another.  Bottom-up: a thread per unvisited vertex looks for a neighbour of
// the last level; rows list the hubs first, so most end at once.
struct BfsShared {
    uint32_t fn, nn;            // frontier, next frontier
    unsigned long long edges;   // row entries of the next frontier
    uint32_t nheavy;
    int32_t heavy[kHeavyList];
};

__device__ void cta_bfs(const Args& A, uint64_t v0, uint64_t v1, BfsShared& S) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint64_t n = v1 - v0;
    for (uint64_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) A.dist[v] = INT_MAX;
    __syncthreads();
    if (threadIdx.x == 0) {
        A.dist[v0] = 0;
        A.q0[v0] = (int32_t)v0;
        S.fn = 1;
        S.edges = A.off[v0 + 1] - A.off[v0];
    }
    __syncthreads();
    int32_t* fq = A.q0 + v0;
    int32_t* nq = A.q1 + v0;
    unsigned long long unexplored = A.off[v1] - A.off[v0];
    bool bottom_up = false;
    auto append = [&](bool won, int32_t v) {
        const unsigned m = __ballot_sync(0xffffffffu, won);
        if (!m) return;
        unsigned long long d = won ? A.off[v + 1] - A.off[v] : 0;
        for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        uint32_t at = 0;
        if (lane == 0) {
            at = atomicAdd(&S.nn, (uint32_t)__popc(m));
            atomicAdd(&S.edges, d);
        }
        at = __shfl_sync(0xffffffffu, at, 0);
        if (won) nq[at + __popc(m & ((1u << lane) - 1u))] = v;
    };
    for (int32_t level = 1;; ++level) {
        const uint32_t fn = S.fn;
        const unsigned long long edges = S.edges;
        __syncthreads();
        if (fn == 0) break;
        unexplored -= edges;
        if (!bottom_up && edges * 15 > unexplored) bottom_up = true;
        else if (bottom_up && (uint64_t)fn * 18 < n) bottom_up = false;
        if (threadIdx.x == 0) {
            S.nn = 0;
            S.edges = 0;
            S.nheavy = 0;
        }
        __syncthreads();
        if (bottom_up) {
            for (uint64_t i = threadIdx.x; i < ((n + 31) & ~31ull); i += blockDim.x) {
                const uint64_t v = v0 + i;
                bool found = false;
                if (i < n && A.dist[v] == INT_MAX) {
                    for (uint64_t j = A.off[v], e = A.off[v + 1]; j < e && !found; ++j)
                        found = A.dist[A.adj[j]] == level - 1;
                    if (found) A.dist[v] = level;
                }
                append(found, (int32_t)v);
            }
        } else {
            auto expand = [&](uint64_t j, uint64_t e) {
                bool won = false;
                int32_t v = 0;
                if (j < e) {
                    v = A.adj[j];
                    if (A.dist[v] == INT_MAX) won = atomicCAS(&A.dist[v], INT_MAX, level) == INT_MAX;
                }
                append(won, v);
            };
            for (uint32_t i = w; i < fn; i += nw) {
                const int32_t u = fq[i];
                const uint64_t b = A.off[u], e = A.off[u + 1];
                if (e - b > kHeavyRow) {
                    uint32_t h = 0;
                    if (lane == 0) h = atomicAdd(&S.nheavy, 1u);
                    h = __shfl_sync(0xffffffffu, h, 0);
                    if (h < kHeavyList) {
                        if (lane == 0) S.heavy[h] = u;
                        continue;
                    }
                }
                for (uint64_t j0 = b; j0 < e; j0 += 32) expand(j0 + lane, e);
            }
            __syncthreads();
            const uint32_t nh = min(S.nheavy, kHeavyList);
            for (uint32_t h = 0; h < nh; ++h) {
                const int32_t u = S.heavy[h];
                const uint64_t b = A.off[u], e = A.off[u + 1];
                for (uint64_t j0 = b + 32 * w; j0 < e; j0 += 32 * nw) expand(j0 + lane, e);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) S.fn = S.nn;
        int32_t* t = fq;
        fq = nq;
        nq = t;
        __syncthreads();
    }
    for (uint64_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
        const int32_t d = A.dist[v];
        A.dist[v] = d == 0 ? -1 : d;  // rank[src] = -1 (src/Graph.cpp:1704)
    }
}

template <int kMode, bool kCopy>
__global__ void __launch_bounds__(kMaxWarps * 32, 2) k_batch(Args A) {
    extern __shared__ uint32_t smem[];
    __shared__ uint32_t s_item;
    __shared__ BfsShared s_bfs;
    while (A.nbfs) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(&A.counter[0], 1u);
        __syncthreads();
        const uint32_t it = s_item;
        if (it >= A.nbfs) break;
        const int32_t g = A.bfs_order[it];
        cta_bfs(A, A.voff[g], A.voff[g + 1], s_bfs);
    }
    if (!A.ntri) return;
    uint32_t* bm = smem + (threadIdx.x >> 5) * kWarpWords(kMode == tc::kCountVertex);
    if constexpr (kCopy) warp_triangles<kMode>(A, A.oriented, bm);
    else warp_triangles<kMode>(A, tc::CsrView{A.off, A.adj, A.dplus, 0}, bm);
}

static uint64_t key_of(uint32_t tasks, int threads, int cps, int order) {
    return ((uint64_t)tasks << 32) | ((uint64_t)threads << 16) | ((uint64_t)cps << 8) | (uint64_t)order;
}

}  // namespace bt
}  // namespace pc

using namespace pc;
using namespace pc::bt;

// The graphs in BFS order: largest first (order 0) or as packed (order 1).
static pc_status batch_build_items(pc_batch* b, uint32_t tasks) {
    std::vector<int32_t> gidx(b->G);
    std::iota(gidx.begin(), gidx.end(), 0);
    if (b->order == 0)
        std::stable_sort(gidx.begin(), gidx.end(), [&](int32_t x, int32_t y) { return b->gm[x] > b->gm[y]; });
    int ntasks = 0;
    for (uint32_t t : {PC_BATCH_TC, PC_BATCH_LCC, PC_BATCH_BFS}) ntasks += (tasks & t) != 0;
    b->nitems = b->G * ntasks;
    PC_TRY(b->items.ensure((size_t)b->G * 4, "batch items"));
    PC_CUDA(cudaMemcpyAsync(b->items.p, gidx.data(), gidx.size() * 4, cudaMemcpyHostToDevice, b->g->stream));
    PC_CUDA(cudaStreamSynchronize(b->g->stream));
    return PC_OK;
}

static pc_status batch_capture(pc_batch* b, uint32_t tasks) {
    const uint64_t key = key_of(tasks, b->threads, b->ctas_per_sm, b->order);
    if (b->exec && b->exec_key == key) return PC_OK;
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    if (b->graph) {
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    PC_TRY(batch_build_items(b, tasks));
    cudaStream_t s = b->g->stream;
    const uint64_t N = b->g->n;
    const bool lcc = tasks & PC_BATCH_LCC, tc = tasks & PC_BATCH_TC;
    Args A;
    A.off = b->g->off.as<uint64_t>();
    A.adj = b->g->adj.as<int32_t>();
    A.voff = b->d_voff.as<uint64_t>();
    A.dplus = b->dplus.as<uint32_t>();
    A.oriented = tc::OrientedView{b->ooff.as<uint32_t>(), b->oids.as<int4>()};
    A.titems = b->titems.as<TriItem>();
    A.ntri = lcc || tc ? b->ntri : 0;
    A.bfs_order = b->items.as<int32_t>();
    A.nbfs = tasks & PC_BATCH_BFS ? b->G : 0;
    A.counter = b->counter.as<uint32_t>();
    A.tc = tc ? b->tc.as<unsigned long long>() : nullptr;
    A.tri = lcc ? b->tri.as<unsigned long long>() : nullptr;
    A.dist = b->dist.as<int32_t>();
    A.q0 = b->q0.as<int32_t>();
    A.q1 = b->q1.as<int32_t>();
    const size_t smem = (size_t)(b->threads / 32) * kWarpWords(lcc) * 4;
    auto kernel = b->oids.p ? (lcc ? k_batch<tc::kCountVertex, true> : k_batch<tc::kCountOnly, true>)
                            : (lcc ? k_batch<tc::kCountVertex, false> : k_batch<tc::kCountOnly, false>);
    PC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const unsigned grid = (unsigned)(sm_count(b->g->device) * b->ctas_per_sm);
    PC_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    cudaMemsetAsync(b->counter.p, 0, 16, s);
    if (tc) cudaMemsetAsync(b->tc.p, 0, (size_t)b->G * 8, s);
    if (lcc) cudaMemsetAsync(b->tri.p, 0, N * 8, s);
    kernel<<<grid, b->threads, smem, s>>>(A);
    if (lcc) k_batch_lcc<<<(unsigned)ceil_div(N, 256), 256, 0, s>>>(A.off, N, A.tri);
    if (tasks & PC_BATCH_TC) cudaMemcpyAsync(b->h_tc, b->tc.p, (size_t)b->G * 8, cudaMemcpyDeviceToHost, s);
    if (tasks & PC_BATCH_LCC) cudaMemcpyAsync(b->h_lcc, b->tri.p, N * 8, cudaMemcpyDeviceToHost, s);
    if (tasks & PC_BATCH_BFS) cudaMemcpyAsync(b->h_bfs, b->dist.p, N * 4, cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamEndCapture(s, &b->graph);
    if (e != cudaSuccess) return cuda_fail(e, "stream capture of the batch launch", __FILE__, __LINE__);
    PC_CUDA(cudaGraphInstantiate(&b->exec, b->graph, 0));
    b->exec_key = key;
    return PC_OK;
}

extern "C" {

pc_status pc_batch_create(const uint64_t* vlist, const int32_t* elist, uint64_t N, uint64_t M, const uint64_t* voff,
                          uint32_t G, pc_batch** out) {
    clear_error();
    if (!out || !voff || G == 0) return fail(PC_ERR_INVALID_INPUT, "bad argument");
    *out = nullptr;
    if (voff[0] != 0 || voff[G] != N) return fail(PC_ERR_INVALID_INPUT, "graph offsets must run from 0 to N");
    for (uint32_t g = 0; g < G; ++g)
        if (voff[g + 1] <= voff[g]) return fail(PC_ERR_INVALID_INPUT, "every graph needs at least one vertex");
    pc_graph* arena = nullptr;
    PC_TRY(pc_graph_create(vlist, elist, nullptr, N, M, 0, &arena));
    pc_batch* b = new pc_batch();
    b->g = arena;
    b->G = G;
    b->voff.assign(voff, voff + G + 1);
    b->gm.resize(G);
    for (uint32_t g = 0; g < G; ++g) b->gm[g] = vlist[voff[g + 1]] - vlist[voff[g]];
    auto bail = [&](pc_status st) {
        const std::string msg = pc_last_error();
        if (b->h_tc) cudaFreeHost(b->h_tc);
        if (b->h_lcc) cudaFreeHost(b->h_lcc);
        if (b->h_bfs) cudaFreeHost(b->h_bfs);
        pc_graph_destroy(b->g);
        delete b;
        return fail(st, msg);
    };
    pc_status st;
    if ((st = b->d_voff.alloc((G + 1) * 8, "graph offsets")) != PC_OK || (st = b->dplus.alloc(N * 4, "dplus")) != PC_OK ||
        (st = b->tri.alloc(N * 8, "triangles per vertex, lcc")) != PC_OK ||
        (st = b->dist.alloc(N * 4, "levels")) != PC_OK || (st = b->q0.alloc(N * 4, "queue")) != PC_OK ||
        (st = b->q1.alloc(N * 4, "queue")) != PC_OK || (st = b->tc.alloc((size_t)G * 8, "counts")) != PC_OK ||
        (st = b->counter.alloc(16, "counter")) != PC_OK)
        return bail(st);
    cudaError_t e = cudaMallocHost(&b->h_tc, (size_t)G * 8);
    if (e == cudaSuccess) e = cudaMallocHost(&b->h_lcc, N * 8);
    if (e == cudaSuccess) e = cudaMallocHost(&b->h_bfs, N * 4);
    if (e == cudaSuccess) e = cudaEventCreate(&b->ev0);
    if (e == cudaSuccess) e = cudaEventCreate(&b->ev1);
    if (e != cudaSuccess) return bail(cuda_fail(e, "pinned staging", __FILE__, __LINE__));
    cudaStream_t s = arena->stream;
    DevBuf chk;
    if ((st = chk.alloc(16, "check")) != PC_OK) return bail(st);
    e = cudaMemcpyAsync(b->d_voff.p, voff, (G + 1) * 8, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(chk.p, 0, 16, s);
    if (e != cudaSuccess) return bail(cuda_fail(e, "batch upload", __FILE__, __LINE__));
    const uint64_t* off = arena->off.as<uint64_t>();
    int32_t *graph_of = b->q0.as<int32_t>(), *base = b->q1.as<int32_t>();
    uint32_t *dplus = b->dplus.as<uint32_t>(), *d_bad = chk.as<uint32_t>(), *d_items = d_bad + 1;
    const unsigned nb = (unsigned)ceil_div(N, 256);
    k_graph_of<<<G, 256, 0, s>>>(b->d_voff.as<uint64_t>(), graph_of, base);
    count_launch();
    k_prepare<<<nb, 256, 0, s>>>(off, arena->adj.as<int32_t>(), b->d_voff.as<uint64_t>(), graph_of, N, dplus, d_bad);
    count_launch();
    k_triangle_items<<<nb, 256, 0, s>>>(off, dplus, graph_of, N, nullptr, d_items);
    count_launch();
    uint32_t chk_h[2] = {0, 0};
    e = cudaMemcpyAsync(chk_h, chk.p, 8, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return bail(cuda_fail(e, "batch preparation", __FILE__, __LINE__));
    if (chk_h[0]) return bail(fail(PC_ERR_INVALID_INPUT, "an edge joins two graphs of the batch"));
    b->ntri = chk_h[1];
    if ((st = b->titems.alloc((size_t)b->ntri * sizeof(TriItem), "triangle items")) != PC_OK) return bail(st);
    e = cudaMemsetAsync(d_items, 0, 4, s);
    if (e != cudaSuccess) return bail(cuda_fail(e, "batch preparation", __FILE__, __LINE__));
    k_triangle_items<<<nb, 256, 0, s>>>(off, dplus, graph_of, N, b->titems.as<TriItem>(), d_items);
    count_launch();
    if (oriented_wanted(N, M, true, arena->device, 0)) {
        // without room for the copy the scans read the CSR
        DevBuf tmp;
        const size_t tb = oriented_temp_bytes(N);
        st = tmp.alloc(tb, "scan scratch");
        if (st == PC_OK)
            st = build_oriented(off, arena->adj.as<int32_t>(), dplus, base, N, M, true, arena->device, s, tmp.p, tb,
                                &b->ooff, &b->oids, &b->ovecs);
        e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) return bail(cuda_fail(e, "batch preparation", __FILE__, __LINE__));
        if (st != PC_OK) {
            b->ooff.release();
            b->oids.release();
            if (st != PC_ERR_OOM) return bail(st);
            clear_error();
        }
    }
    e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return bail(cuda_fail(e, "batch preparation", __FILE__, __LINE__));
    *out = b;
    return PC_OK;
}

pc_status pc_batch_destroy(pc_batch* b) {
    if (!b) return PC_OK;
    cudaSetDevice(b->g->device);
    cudaStreamSynchronize(b->g->stream);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    if (b->ev0) cudaEventDestroy(b->ev0);
    if (b->ev1) cudaEventDestroy(b->ev1);
    if (b->h_tc) cudaFreeHost(b->h_tc);
    if (b->h_lcc) cudaFreeHost(b->h_lcc);
    if (b->h_bfs) cudaFreeHost(b->h_bfs);
    pc_graph* g = b->g;
    delete b;
    return pc_graph_destroy(g);
}

pc_status pc_batch_set_schedule(pc_batch* b, int32_t threads, int32_t ctas_per_sm, int32_t order) {
    clear_error();
    if (!b) return fail(PC_ERR_INVALID_INPUT, "null batch");
    if ((threads != 256 && threads != 512) || ctas_per_sm < 1 || ctas_per_sm > 4 || (order != 0 && order != 1))
        return fail(PC_ERR_INVALID_INPUT, "schedule: threads 256|512, ctas_per_sm 1..4, order 0|1");
    b->threads = threads;
    b->ctas_per_sm = ctas_per_sm;
    b->order = order;
    return PC_OK;
}

pc_status pc_batch_run(pc_batch* b, uint32_t tasks, uint64_t* tc, double* lcc, int32_t* bfs, pc_batch_stats* stats) {
    clear_error();
    if (!b || !tasks || (tasks & ~7u)) return fail(PC_ERR_INVALID_INPUT, "bad argument");
    if (((tasks & PC_BATCH_TC) && !tc) || ((tasks & PC_BATCH_LCC) && !lcc) || ((tasks & PC_BATCH_BFS) && !bfs))
        return fail(PC_ERR_INVALID_INPUT, "missing output buffer");
    PC_TRY(use_device(b->g));
    PC_TRY(batch_capture(b, tasks));
    cudaStream_t s = b->g->stream;
    PC_CUDA(cudaEventRecord(b->ev0, s));
    PC_CUDA(cudaGraphLaunch(b->exec, s));
    PC_CUDA(cudaEventRecord(b->ev1, s));
    PC_CUDA(cudaStreamSynchronize(s));
    PC_CUDA(cudaGetLastError());
    count_launch();
    const uint64_t N = b->g->n;
    if (tasks & PC_BATCH_TC) memcpy(tc, b->h_tc, (size_t)b->G * 8);
    if (tasks & PC_BATCH_LCC) memcpy(lcc, b->h_lcc, N * 8);
    if (tasks & PC_BATCH_BFS) memcpy(bfs, b->h_bfs, N * 4);
    if (stats) {
        float ms = 0.f;
        PC_CUDA(cudaEventElapsedTime(&ms, b->ev0, b->ev1));
        stats->ms = ms;
        stats->items = b->nitems;
        stats->threads = b->threads;
        stats->ctas_per_sm = b->ctas_per_sm;
        stats->order = b->order;
    }
    return PC_OK;
}

pc_status pc_batch_autotune(pc_batch* b, uint32_t tasks, pc_batch_stats* best) {
    clear_error();
    if (!b) return fail(PC_ERR_INVALID_INPUT, "null batch");
    const uint64_t N = b->g->n;
    std::vector<uint64_t> tc(b->G);
    std::vector<double> lcc(N);
    std::vector<int32_t> bfs(N);
    double best_ms = 1e30;
    int bt = b->threads, bc = b->ctas_per_sm, bo = b->order;
    const int thr[] = {256, 512};
    for (int t : thr)
        for (int c = 1; c <= 4; c *= 2)
            for (int o = 0; o < 2; ++o) {
                if (t == 512 && c > 2) continue;
                PC_TRY(pc_batch_set_schedule(b, t, c, o));
                pc_batch_stats st;
                PC_TRY(pc_batch_run(b, tasks, tc.data(), lcc.data(), bfs.data(), &st));  // warm / capture
                PC_TRY(pc_batch_run(b, tasks, tc.data(), lcc.data(), bfs.data(), &st));
                if (st.ms < best_ms) {
                    best_ms = st.ms;
                    bt = t;
                    bc = c;
                    bo = o;
                }
            }
    PC_TRY(pc_batch_set_schedule(b, bt, bc, bo));
    if (best) {
        PC_TRY(pc_batch_run(b, tasks, tc.data(), lcc.data(), bfs.data(), best));
    }
    return PC_OK;
}

}  // extern "C"
