// Frontier algorithms: BFS, SSSP, PageRank, k-core, MIS, CDLP (sm_100a).
//
// All kernels work on the symmetric CSR in the internal id space; inputs and
// outputs are mapped to the caller's id space (identity unless the view was
// reordered).  Frontiers are compacted queues; appends are warp-aggregated
// (one atomic per warp and step).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "grid_sync.cuh"
#include "pc_internal.cuh"
#include "synth_rng.h"
#include "tile_expand.cuh"

namespace pc {
namespace fr {

constexpr int kThreads = 256;
constexpr int32_t kInf = INT_MAX;
// k-core: ids below this have their degree decrements gathered per CTA
constexpr int kKcoreHubs = 4096;
constexpr int kKcoreThreads = 512;       // k-core: threads per CTA
constexpr int kKcorePerSm = 2;
constexpr uint32_t kLocalQ = 2048;       // ... its queue of claimed vertices
constexpr uint32_t kLocalEdges = 16384;  // ... peeled by the CTA itself while their rows stay below this
constexpr int kLocalRounds = 1 << 14;    // ... for so many rounds a step, while the others wait
constexpr size_t kKcoreSmem = 80 * 1024;
static_assert(kKcoreHubs % kKcoreThreads == 0, "the flush loop needs a uniform trip count");

// Appends `val` for every lane with pred set; all 32 lanes of the warp must
// call it together.
__device__ __forceinline__ void warp_append(bool pred, int32_t val, int32_t* __restrict__ q,
                                            uint32_t* __restrict__ qn) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(qn, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (pred) q[base + __popc(m & ((1u << lane) - 1u))] = val;
}

__device__ __forceinline__ uint64_t warp_sum_u64(uint64_t x) {
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Pull sweeps (PageRank, CDLP): lanes of a short row (4 lanes measured 10 %
// faster than 8 for PageRank at RMAT-22, 16 lanes 16 % slower).
constexpr int kPullLanes = 4;

// ---- BFS -------------------------------------------------------------------

// Direction-optimising (Beamer, Asanovic, Patterson, SC'12) in one persistent
// kernel, a grid barrier per level: top-down levels expand the frontier's
// queues (tx::expand); bottom-up levels look for a neighbour of the last
// level at every unvisited vertex and only count what they find.  Back from
// bottom-up, one step collects the frontier's queues from the levels.
// The state lives in three rotating records (see KState).
//
// Bound at RMAT-22: the copy of the levels to the host (0.3 of 0.6 ms), then
// the dependent loads of seven levels and their barriers.  With two launches
// and a host read per level, and a warp per row, 0.76-0.97 ms; ER-20 0.47 ->
// 0.25 ms, RMAT-16 0.32 -> 0.14, RMAT-10 0.18 -> 0.06.
struct __align__(16) BfsState {
    uint32_t nl, nh;      // the frontier's queues (queued)
    uint32_t fn;          // vertices in the frontier
    int32_t level;        // of the frontier's unvisited neighbours
    uint64_t edges;       // row entries of the frontier
    uint64_t unexplored;  // ... and of it and every later vertex
    int32_t bottom_up;    // direction of the level before
    int32_t queued;       // the frontier is in the queues; 2: and top-down is decided
    int32_t par;          // queues in use
    int32_t pad;
};

__global__ void k_bfs_init(const uint64_t* __restrict__ off, uint64_t n, uint64_t m, int32_t src,
                           int32_t* __restrict__ dist, tx::Queues Q, BfsState* S) {
    for (uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < n; u += (uint64_t)gridDim.x * blockDim.x)
        dist[u] = u == (uint64_t)src ? 0 : kInf;
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        if (threadIdx.x < 3)
            S[threadIdx.x] = BfsState{0, 0, threadIdx.x == 0, 1, threadIdx.x ? 0 : off[src + 1] - off[src], m, 0, 1, 0, 0};
        __syncwarp();
        tx::enqueue<1>(&src, threadIdx.x == 0, off, Q, &S[0].nl, &S[0].nh);
    }
}

__global__ void __launch_bounds__(tx::kThreads, 6)
    k_bfs_persistent(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj, uint64_t n, int32_t src,
                     int32_t* dist, tx::Queues q0, tx::Queues q1, BfsState* S, GridBarrier* gb, uint64_t max_steps,
                     uint64_t limit_ns) {
    __shared__ tx::Tile s_tile[tx::kWarps];
    __shared__ tx::Buffer s_buf[tx::kWarps];
    __shared__ unsigned long long s_edges;
    __shared__ uint32_t s_fn;
    tx::Tile& T = s_tile[threadIdx.x >> 5];
    tx::Buffer& B = s_buf[threadIdx.x >> 5];
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    const int lane = threadIdx.x & 31;
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t nr = (n + 127) & ~127ull;  // whole warps of four vertices a lane
    // levels of vertices v .. v + 3 (v a multiple of 4; -2 past the last one)
    auto levels4 = [&](uint64_t v) {
        if (v + 4 <= n) return __ldcg(reinterpret_cast<const int4*>(dist + v));
        int4 d = make_int4(-2, -2, -2, -2);
        if (v < n) d.x = __ldcg(dist + v);
        if (v + 1 < n) d.y = __ldcg(dist + v + 1);
        if (v + 2 < n) d.z = __ldcg(dist + v + 2);
        return d;
    };
    if (threadIdx.x == 0) {
        s_edges = 0;
        s_fn = 0;
    }
    __syncthreads();
    uint64_t step = 0;
    for (; step < max_steps; ++step) {
        const BfsState* in = &S[step % 3];
        BfsState* out = &S[(step + 1) % 3];
        const uint32_t nl = __ldcg(&in->nl), nh = __ldcg(&in->nh), fn = __ldcg(&in->fn);
        const int32_t level = __ldcg(&in->level), queued = __ldcg(&in->queued), par = __ldcg(&in->par);
        const uint64_t edges = __ldcg(&in->edges), unexplored = __ldcg(&in->unexplored) - edges;
        // every CTA reads the same record, so all leave at the same step
        if (fn == 0) break;
        const int32_t was = __ldcg(&in->bottom_up);
        const bool bottom_up = queued != 2 && (was ? fn * 18ull >= n : edges * 15 > unexplored);
        const bool collect = !bottom_up && !queued;  // the frontier is not in the queues
        // A level that expands a good part of what is left finds most of the
        // graph, and the next one runs bottom-up: it is counted, not queued
        // (RMAT-22, 0.8 M vertices found: 130 us for the level with queues).
        const bool many = !bottom_up && !collect && edges * 64 > unexplored;
        if (lead) {
            BfsState* clr = &S[(step + 2) % 3];
            clr->nl = clr->nh = clr->fn = 0;
            clr->edges = 0;
            out->bottom_up = bottom_up;
            out->queued = collect ? 2 : !bottom_up && !many;
            out->par = bottom_up ? par : 1 - par;
            out->level = collect ? level : level + 1;
            out->unexplored = collect ? unexplored + edges : unexplored;
            if (collect) {
                out->fn = fn;
                out->edges = edges;
            }
        }
        const tx::Queues& Q = par ? q1 : q0;
        const tx::Queues& QN = par ? q0 : q1;
        uint64_t found_edges = 0;
        uint32_t found = 0;
        if (collect) {
            uint32_t nb = 0;
            for (uint64_t v = 4 * tid; v < nr; v += 4 * stride) {
                const int4 d = levels4(v);
                tx::find(B, nb, d.x == level - 1, (int32_t)v);
                tx::find(B, nb, d.y == level - 1, (int32_t)v + 1);
                tx::find(B, nb, d.z == level - 1, (int32_t)v + 2);
                tx::find(B, nb, d.w == level - 1, (int32_t)v + 3);
                if (nb > tx::kBuf - 128) tx::flush(B, nb, off, QN, &out->nl, &out->nh);
            }
            tx::flush(B, nb, off, QN, &out->nl, &out->nh);
        } else if (bottom_up) {
            // (four vertices a thread with their loads together: a quarter
            // slower; the rows that go on then wait for one another)
            // The plain loads of the neighbours' levels see all of the last
            // step's (grid_sync); this step's, old or new, are not looked for.
            for (uint64_t v = tid; v < n; v += stride) {
                if (__ldcg(dist + v) != kInf) continue;
                const uint64_t b = off[v], e = off[v + 1];
                bool hit = false;
                // four ids a load; the ids outside [b, e) are not looked at
                for (uint64_t q = b & ~3ull; q < e && !hit; q += 4) {
                    const int4 a = __ldg(reinterpret_cast<const int4*>(adj + q));
                    hit = (q >= b && dist[a.x] == level - 1) || (q + 1 >= b && q + 1 < e && dist[a.y] == level - 1) ||
                          (q + 2 >= b && q + 2 < e && dist[a.z] == level - 1) || (q + 3 < e && dist[a.w] == level - 1);
                }
                if (hit) {
                    dist[v] = level;
                    found_edges += e - b;
                    ++found;
                }
            }
        } else {
            uint32_t nb = 0;
            tx::expand(
                T, off, Q, nl, nh, [](int32_t) { return 0; },
                [&](const uint64_t* j, const int32_t*, const bool* ok) {
                    int32_t v[tx::kPerLane];
                    bool open[tx::kPerLane];
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) v[k] = ok[k] ? __ldcs(adj + j[k]) : 0;
                    // a level read here may be an old "unvisited" from L1: atomicCAS decides
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) open[k] = ok[k] && dist[v[k]] == kInf;
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k)
                        open[k] = open[k] && atomicCAS(&dist[v[k]], kInf, level) == kInf;
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) {
                        if (many) found_edges += open[k] ? off[v[k] + 1] - off[v[k]] : 0;
                        else tx::find(B, nb, open[k], v[k]);
                        found += open[k];
                    }
                },
                [&]() {
                    if (nb > tx::kBuf - tx::kRound) found_edges += tx::flush(B, nb, off, QN, &out->nl, &out->nh);
                });
            found_edges += tx::flush(B, nb, off, QN, &out->nl, &out->nh);
        }
        found_edges = warp_sum_u64(found_edges);
        found = __reduce_add_sync(0xffffffffu, found);
        if (lane == 0 && found) {
            atomicAdd(&s_edges, (unsigned long long)found_edges);
            atomicAdd(&s_fn, found);
        }
        __syncthreads();
        if (threadIdx.x == 0 && s_fn) {
            atomicAdd((unsigned long long*)&out->edges, s_edges);
            atomicAdd(&out->fn, s_fn);
            s_edges = 0;
            s_fn = 0;
        }
        if (!grid_sync(gb, limit_ns)) return;
    }
    if (lead) {
        dist[src] = -1;  // rank[src] = -1 (src/Graph.cpp:1704)
        if (step == max_steps) atomicExch(&gb->err, 2);
    }
}

// ---- SSSP: frontier Bellman-Ford and delta-stepping --------------------------
//
// Both forms relax the rows of a frontier with atomicMin and queue every
// vertex whose distance falls; they differ in which improved vertices are
// relaxed next.  Bellman-Ford (an unbounded bucket) relaxes all of them in the
// next step.  Delta-stepping (Meyer and Sanders, "Delta-stepping: a
// parallelizable shortest path algorithm", J. Algorithms 2003, in the
// near/far-pile form of Davidson, Baxter, Garland and Owens, IPDPS 2014)
// relaxes only vertices whose new distance is below the current bucket's
// upper bound `thr` ("near"); the others go to a far pile that is split when
// the bucket is exhausted.  Both are label-correcting: every improvement is
// queued, so both end at the exact shortest distances (integer weights >= 0).
//
// One persistent kernel runs all steps, a grid barrier between them, so a
// bucket costs microseconds instead of launches and host reads, and narrow
// buckets, which relax fewer edges in vain, pay.  A step is a relaxation of
// the near frontier (tx::expand) or, when that is empty, the split of the far
// pile.  Steps keep their state in three rotating records (see KState).
//
// Bound at RMAT-22 (6.6 -> 2.2 ms a call, 0.3 ms of it the copy back): the
// gathers of the neighbours' distances, 2.9 m of them, from L1 and L2.  Small
// graphs: barriers and chains of atomics, 4-10 us a step (RMAT-16 0.90 -> 0.37
// ms, RMAT-10 0.50 -> 0.15); ER-20 5.2 -> 0.92 ms.
struct __align__(16) SsspState {
    uint32_t nl, nh;  // near queues' lengths
    int32_t thr;      // near bound (exclusive)
    int32_t par;      // near queues in use
    int32_t splits;   // splits so far: the far pile is far[splits % 2], its counters those of splits % 3
    int32_t pad[3];
};
struct SsspFar {
    uint32_t n[3];
    int32_t min[3];  // a bound on the pile's smallest distance
};

// dist, stamps and flags cleared; the source queued.
__global__ void k_sssp_init(const uint64_t* __restrict__ off, uint64_t n, int32_t src, int32_t bound,
                            const int32_t* __restrict__ delta, int32_t* __restrict__ dist, int32_t* __restrict__ stamp,
                            int32_t* __restrict__ farflag, tx::Queues Q, SsspState* S, SsspFar* F) {
    for (uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < n; u += (uint64_t)gridDim.x * blockDim.x) {
        dist[u] = u == (uint64_t)src ? 0 : INT_MAX / 2;  // src/test.cpp:202-203
        stamp[u] = 0;
        farflag[u] = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        if (threadIdx.x < 3) {
            S[threadIdx.x] = SsspState{0, 0, bound ? bound : *delta, 0, 0, {0, 0, 0}};
            F->n[threadIdx.x] = 0;
            F->min[threadIdx.x] = INT_MAX;
        }
        __syncwarp();
        tx::enqueue<1>(&src, threadIdx.x == 0, off, Q, &S[0].nl, &S[0].nh);
    }
}

// The width chosen by the library (any width gives the same distances): the
// mean of up to 2^16 weights taken at equal steps.  A step costs about 8 us
// (barrier and one chain of dependent loads), and the wider a bucket, the more
// edges are relaxed in vain.  Measured with weights 1..255 (mean 128), ms at
// widths of 64 / 128 / 256 / 1024: RMAT-22 2.60 / 2.56 / 2.67 / 2.57, RMAT-18
// 0.81 / 0.69 / 0.66 / 0.61, ER-20 1.64 / 1.36 / 1.92 / 2.08 (with a dearer
// step than now).  One CTA.
__global__ void k_sssp_delta(const int32_t* __restrict__ w, uint64_t m, int32_t* __restrict__ delta) {
    __shared__ unsigned long long sum;
    if (threadIdx.x == 0) sum = 0;
    __syncthreads();
    const uint64_t step = m > 65536 ? m / 65536 : 1, cnt = (m + step - 1) / step;
    unsigned long long x = 0;
    for (uint64_t i = threadIdx.x; i < cnt; i += blockDim.x) x += (unsigned long long)(uint32_t)w[i * step];
    x = warp_sum_u64(x);
    if ((threadIdx.x & 31) == 0) atomicAdd(&sum, x);
    __syncthreads();
    if (threadIdx.x == 0) {
        const double mean = cnt ? (double)sum / (double)cnt : 1.0;
        *delta = (int32_t)fmin((double)(1 << 30), fmax(1.0, round(mean)));
    }
}

__global__ void __launch_bounds__(tx::kThreads, 5)
    k_sssp_persistent(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj, const int32_t* __restrict__ w,
                      int32_t* dist, int32_t* stamp, int32_t* farflag, tx::Queues q0, tx::Queues q1, int32_t* far0,
                      int32_t* far1, const int32_t* __restrict__ chosen, int32_t given, SsspState* S, SsspFar* F,
                      GridBarrier* gb, uint64_t max_steps, uint64_t limit_ns) {
    __shared__ tx::Tile s_tile[tx::kWarps];
    __shared__ tx::Buffer s_near[tx::kWarps], s_far[tx::kWarps];
    const int32_t delta = chosen ? *chosen : given;
    tx::Tile& T = s_tile[threadIdx.x >> 5];
    tx::Buffer& near_buf = s_near[threadIdx.x >> 5];
    tx::Buffer& far_buf = s_far[threadIdx.x >> 5];
    uint32_t nnear = 0, nfound_far = 0;
    int32_t far_min = INT_MAX;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    const int lane = threadIdx.x & 31;
    auto flush_far = [&](int32_t* far, int c) {
        if (nfound_far == 0) return;
        __syncwarp();
        uint32_t at = 0;
        if (lane == 0) at = atomicAdd(&F->n[c], nfound_far);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (uint32_t i = lane; i < nfound_far; i += 32) far[at + i] = far_buf.v[i];
        __syncwarp();
        nfound_far = 0;
    };
    auto flush_far_min = [&](int c) {
        const int32_t mn = __reduce_min_sync(0xffffffffu, far_min);
        if (lane == 0 && mn != INT_MAX) atomicMin(&F->min[c], mn);
        far_min = INT_MAX;
    };
    uint64_t step = 0;
    for (; step < max_steps; ++step) {
        const SsspState* in_p = &S[step % 3];
        const int4 r0 = __ldcg(reinterpret_cast<const int4*>(in_p));
        const uint32_t nl = (uint32_t)r0.x, nh = (uint32_t)r0.y;
        const int32_t thr = r0.z, par = r0.w, splits = __ldcg(&in_p->splits);
        SsspState* out = &S[(step + 1) % 3];
        const int c = splits % 3;
        int32_t* far = splits & 1 ? far1 : far0;
        const bool relax = nl || nh;
        const uint32_t nfar = relax ? 0u : __ldcg(&F->n[c]);
        // every CTA reads the same record, so all leave at the same step
        if (!relax && nfar == 0) break;
        if (lead) {
            SsspState* clr = &S[(step + 2) % 3];
            clr->nl = clr->nh = 0;
            out->par = 1 - par;
        }
        const tx::Queues& Q = par ? q1 : q0;
        const tx::Queues& QN = par ? q0 : q1;
        const int32_t mark = (int32_t)step + 1;  // stamp of the vertices queued in this step
        if (relax) {
            if (lead) {
                out->thr = thr;
                out->splits = splits;
            }
            tx::expand(
                T, off, Q, nl, nh, [&](int32_t u) { return __ldcg(dist + u); },
                [&](const uint64_t* j, const int32_t* du, const bool* ok) {
                    int32_t v[tx::kPerLane], nd[tx::kPerLane];
                    bool better[tx::kPerLane];
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) {
                        v[k] = ok[k] ? __ldcs(adj + j[k]) : 0;
                        nd[k] = ok[k] ? du[k] + __ldcs(w + j[k]) : INT_MAX;
                    }
                    // A distance read here may be an older, larger one from L1:
                    // atomicMin decides (reading L2 each time: 3.9 instead of
                    // 2.6 ms at RMAT-22, the hubs' distances are hot).  Each
                    // kind of access is issued for all edges before the first
                    // answer is needed.
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) better[k] = nd[k] < dist[v[k]];
                    if (!__any_sync(0xffffffffu, better[0] || better[1] || better[2] || better[3])) return;
                    int32_t old[tx::kPerLane];
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) old[k] = better[k] ? atomicMin(&dist[v[k]], nd[k]) : INT_MIN;
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) {
                        better[k] = nd[k] < old[k];
                        old[k] = better[k] ? atomicExch(nd[k] < thr ? &stamp[v[k]] : &farflag[v[k]], nd[k] < thr ? mark : 1)
                                           : 0;
                    }
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) {
                        const bool near = better[k] && nd[k] < thr && old[k] != mark;
                        const bool away = better[k] && nd[k] >= thr && old[k] == 0;
                        tx::find(near_buf, nnear, near, v[k]);
                        tx::find(far_buf, nfound_far, away, v[k]);
                        if (away) far_min = min(far_min, nd[k]);
                    }
                },
                [&]() {
                    if (nnear > tx::kBuf - tx::kRound) tx::flush(near_buf, nnear, off, QN, &out->nl, &out->nh);
                    if (nfound_far > tx::kBuf - tx::kRound) flush_far(far, c);
                });
            tx::flush(near_buf, nnear, off, QN, &out->nl, &out->nh);
            flush_far(far, c);
            flush_far_min(c);
        } else {
            // Split of the far pile at the next bucket [thr, hi): entries whose
            // distance fell below thr were relaxed when it fell and are
            // dropped; entries below hi become the near frontier; the rest
            // go to the other pile.  Empty buckets are skipped.
            const int32_t mn = max(__ldcg(&F->min[c]), thr);
            const int32_t hi = (int32_t)min((int64_t)INT_MAX, (int64_t)mn + delta);
            const int c2 = (splits + 1) % 3, c3 = (splits + 2) % 3;
            int32_t* far2 = splits & 1 ? far0 : far1;
            if (lead) {
                out->thr = hi;
                out->splits = splits + 1;
                F->n[c3] = 0;  // last read in the split before, next written in the one after
                F->min[c3] = INT_MAX;
            }
            const uint32_t gw = blockIdx.x * tx::kWarps + (threadIdx.x >> 5), nw = gridDim.x * tx::kWarps;
            for (uint64_t i0 = gw * 32ull; i0 < nfar; i0 += nw * 32ull) {
                const uint64_t i = i0 + lane;
                bool near = false, keep = false;
                int32_t v = 0;
                if (i < nfar) {
                    v = __ldcg(far + i);
                    const int32_t d = __ldcg(dist + v);
                    keep = d >= hi;
                    if (!keep) {
                        farflag[v] = 0;
                        near = d >= thr;
                    } else {
                        far_min = min(far_min, d);
                    }
                }
                tx::find(near_buf, nnear, near, v);
                tx::find(far_buf, nfound_far, keep, v);
                if (nnear > tx::kBuf - 32) tx::flush(near_buf, nnear, off, QN, &out->nl, &out->nh);
                if (nfound_far > tx::kBuf - 32) flush_far(far2, c2);
            }
            tx::flush(near_buf, nnear, off, QN, &out->nl, &out->nh);
            flush_far(far2, c2);
            flush_far_min(c2);
        }
        if (!grid_sync(gb, limit_ns)) return;
    }
    if (lead && step == max_steps) atomicExch(&gb->err, 2);
}

// ---- k-core ----------------------------------------------------------------------

// Device-driven peeling in one persistent kernel.  A step either scans the
// remaining vertices at the next level or peels the frontier that an earlier
// step of the level left in the queues; a grid barrier separates steps.
//
// Within a level the order of peeling does not matter, so a CTA peels what it
// finds at once: vertices that the scan or a decrement takes below the level
// go to the CTA's own queue, whose rows it lays end to end (a block scan) and
// takes kPerLane entries per thread at a time, round after round until the
// queue is dry.  A vertex is claimed by the compare-and-swap that sets its
// core number, since the scan and the decrements of other CTAs may meet at
// it.  What does not fit the queue, or would keep one CTA busy for long (rows
// of more than `local_edges` entries together), goes to the next step's queues,
// which all CTAs share (tx::expand).  So most levels take one step.
//
// A chain peels one vertex a round (2.7 us).  After kLocalRounds rounds a CTA
// leaves the rest of its queue for itself in the next step, so that a step keeps
// the others at the barrier for tens of milliseconds, not for seconds.  With 1024
// rounds CTAs of unequal rounds waited for one another too often (a grid of 700
// x 700 vertices 7.0 instead of 4.7 ms); through the shared queues, chains from
// both ends of a path came into one CTA, where the gathered decrements of the one
// waited for the other's end (20 K vertices: 49 instead of 29 ms).
//
// The state lives in three rotating records: step i reads S[i % 3],
// accumulates into S[(i+1) % 3] (counters cleared by step i-1) and clears
// S[(i+2) % 3], which no CTA reads during step i.  Core numbers are read
// through L1, which may hold an old "unpeeled": the entry then decrements a
// peeled vertex's degree, which nobody looks at any more.
//
// Bound (RMAT-22): latency.  The 128 M entries are read once, but in some 300
// dependent steps of a barrier and, per cascade round, one chain of row, id,
// core number and decrement.  16.6 -> 8.5 ms a call (RMAT-16 3.2 -> 2.2, ER-20
// 1.6 -> 0.88) against a step per scan and per round of spilled rows, with a
// warp per row.  CTAs of 256 / 512 / 1024 threads, 1024 threads an SM: 9.0 /
// 8.5 / 9.9 ms; local_edges of 4 K / 16 K / 64 K: 9.2 / 8.5 / 10.7 ms.
struct __align__(16) KState {
    uint32_t nl, nh;   // the frontier's queues
    uint32_t rn;       // vertices on the remaining list
    int32_t ml;        // minimum degree kept by a scan
    int32_t k;         // level of the step that wrote this record
    int32_t par;       // frontier queues in use
    int32_t rpar;      // remaining list in use
    int32_t dirty;     // whether the level claimed vertices before this step
    uint32_t claimed;  // vertices the step claimed
    int32_t top;       // largest core number before this step
    uint32_t rest;     // CTAs that left a rest of their own queue for the step that reads the record
    int32_t pad;
};

__global__ void k_kcore_init(const uint64_t* __restrict__ off, uint64_t n, int32_t* __restrict__ deg,
                             int32_t* __restrict__ core, int32_t* __restrict__ rem, KState* S, int32_t* d_top,
                             GridBarrier* gb) {
    const uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (u < 3) S[u] = KState{0, 0, u ? 0u : (uint32_t)n, INT_MAX, 0, 0, 0, 1, 0, 0, 0, 0};
    if (u == 0) {
        *d_top = 0;
        *gb = GridBarrier{};
    }
    if (u >= n) return;
    deg[u] = (int32_t)(off[u + 1] - off[u]);
    core[u] = -1;
    rem[u] = (int32_t)u;
}

struct KcoreTile {
    uint64_t base[kKcoreThreads];
    uint32_t start[kKcoreThreads];
};

__global__ void __launch_bounds__(kKcoreThreads, kKcorePerSm) k_kcore_persistent(
    const uint64_t* __restrict__ off, const int32_t* __restrict__ adj, uint64_t n, int32_t* deg, int32_t* core,
    int32_t* rem0, int32_t* rem1, tx::Queues q0, tx::Queues q1, KState* S, GridBarrier* gb, uint64_t max_steps,
    uint64_t limit_ns, int32_t* d_top, uint32_t local_edges) {
    constexpr int kWarps = kKcoreThreads / 32;
    extern __shared__ __align__(16) unsigned char kcore_smem[];
    struct Smem {
        KcoreTile tile;                 // the local queue's rows
        tx::Tile warp_tile[kWarps];     // tx::expand
        tx::Buffer spill[kWarps];       // for the next step's queues
        tx::Buffer keep[kWarps];        // for the remaining list
        int32_t lq[2][kLocalQ];         // the CTA's own queue, two rounds
        int32_t dec[kKcoreHubs];        // decrements of the lowest ids (the hubs, once ids are degree-ordered)
        uint32_t warp_sum[kWarps];
        uint32_t lqn[2];                // entries offered (those past kLocalQ went to spill)
        uint32_t claimed;
        int32_t ml;
        int any_dec;
    };
    static_assert(sizeof(Smem) <= kKcoreSmem, "dynamic shared memory of the launch");
    Smem& M = *reinterpret_cast<Smem*>(kcore_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    for (int i = threadIdx.x; i < kKcoreHubs; i += kKcoreThreads) M.dec[i] = 0;
    if (threadIdx.x == 0) {
        M.lqn[0] = M.lqn[1] = 0;
        M.claimed = 0;
        M.ml = INT_MAX;
        M.any_dec = 0;
    }
    __syncthreads();
    tx::Buffer& spill = M.spill[warp];
    tx::Buffer& keep = M.keep[warp];
    uint32_t nspill = 0, nkeep = 0;
    int rd = 0;  // the CTA's queue in use, which may hold a rest of the step before
    uint64_t step = 0;
    for (; step < max_steps; ++step) {
        const KState* in = &S[step % 3];
        KState* out = &S[(step + 1) % 3];
        const int4 r0 = __ldcg(reinterpret_cast<const int4*>(in));
        const int4 r1 = __ldcg(reinterpret_cast<const int4*>(in) + 1);
        const int4 r2 = __ldcg(reinterpret_cast<const int4*>(in) + 2);
        const uint32_t nl = (uint32_t)r0.x, nh = (uint32_t)r0.y, rn = (uint32_t)r0.z;
        const int32_t par = r1.y, rpar = r1.z;
        const bool peel = nl || nh || r2.z;
        const bool dirty = r1.w || r2.x;  // the level of the last step claimed something
        const int32_t k = peel ? r1.x : (dirty || r0.w == INT_MAX ? r1.x + 1 : max(r1.x + 1, r0.w + 1));
        const int32_t top = r2.x ? max(r2.y, r1.x - 1) : r2.y;
        // every CTA reads the same record, so all leave at the same step
        if (!peel && (rn == 0 || (uint64_t)k >= n)) {
            // vertices never peeled (only in a complete graph) keep core 0
            if (rn)
                for (uint64_t u = blockIdx.x * (uint64_t)kKcoreThreads + threadIdx.x; u < n;
                     u += (uint64_t)gridDim.x * kKcoreThreads)
                    if (__ldcg(core + u) < 0) core[u] = 0;
            if (lead) *d_top = top;
            return;
        }
        if (lead) {
            KState* clr = &S[(step + 2) % 3];
            clr->nl = clr->nh = clr->rn = clr->claimed = clr->rest = 0;
            clr->ml = INT_MAX;
            if (peel) out->rn = rn;  // a peel step keeps the remaining list
            out->k = k;
            out->par = 1 - par;
            out->rpar = peel ? rpar : 1 - rpar;
            out->dirty = peel && dirty;
            out->top = top;
        }
        const tx::Queues& Q = par ? q1 : q0;
        const tx::Queues& QN = par ? q0 : q1;
        uint32_t claimed = 0;
        // a claimed vertex whose row is to be peeled, for every lane with pred set
        auto push = [&](bool pred, int32_t v, int wr) {
            const unsigned m = __ballot_sync(0xffffffffu, pred);
            if (!m) return;
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&M.lqn[wr], (uint32_t)__popc(m));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
            if (pred && at < kLocalQ) M.lq[wr][at] = v;
            if (__any_sync(0xffffffffu, pred && at >= kLocalQ)) {
                tx::find(spill, nspill, pred && at >= kLocalQ, v);
                if (nspill > tx::kBuf - 32) tx::flush(spill, nspill, off, QN, &out->nl, &out->nh);
            }
        };
        auto claim = [&](int32_t v) { return atomicCAS(&core[v], -1, k - 1) == -1; };
        // kPerLane entries of peeled rows; each kind of access is issued for
        // all of them before the first answer is needed
        auto peel_entries = [&](const uint64_t* j, const bool* ok, int wr) {
            int32_t v[tx::kPerLane], old[tx::kPerLane];
            bool open[tx::kPerLane];
#pragma unroll
            for (int i = 0; i < tx::kPerLane; ++i) v[i] = ok[i] ? __ldcs(adj + j[i]) : 0;
#pragma unroll
            for (int i = 0; i < tx::kPerLane; ++i) open[i] = ok[i] && core[v[i]] < 0;
#pragma unroll
            for (int i = 0; i < tx::kPerLane; ++i) {
                old[i] = 0;
                if (!open[i]) continue;
                if (v[i] < kKcoreHubs) {
                    atomicAdd(&M.dec[v[i]], 1);
                    M.any_dec = 1;
                } else {
                    old[i] = atomicSub(&deg[v[i]], 1);
                }
            }
#pragma unroll
            for (int i = 0; i < tx::kPerLane; ++i) {
                const bool won = open[i] && old[i] == k && claim(v[i]);
                claimed += won;
                push(won, v[i], wr);
            }
        };
        if (peel) {
            tx::expand(
                M.warp_tile[warp], off, Q, nl, nh, [](int32_t) { return 0; },
                [&](const uint64_t* j, const int32_t*, const bool* ok) { peel_entries(j, ok, rd); }, []() {});
        } else {
            const int32_t* rem = rpar ? rem1 : rem0;
            int32_t* rem2 = rpar ? rem0 : rem1;
            auto flush_keep = [&]() {
                if (nkeep == 0) return;
                __syncwarp();
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(&out->rn, nkeep);
                at = __shfl_sync(0xffffffffu, at, 0);
                for (uint32_t i = lane; i < nkeep; i += 32) rem2[at + i] = keep.v[i];
                __syncwarp();
                nkeep = 0;
            };
            int32_t mn = INT_MAX;
            const uint64_t nr = ((uint64_t)rn + 31) & ~(uint64_t)31;
            for (uint64_t i = blockIdx.x * (uint64_t)kKcoreThreads + threadIdx.x; i < nr;
                 i += (uint64_t)gridDim.x * kKcoreThreads) {
                bool pl = false, stay = false;
                int32_t u = 0;
                if (i < rn) {
                    u = __ldcg(rem + i);
                    const int32_t c = __ldcg(core + u), d = __ldcg(deg + u);
                    if (c < 0) {
                        if (d >= k) {
                            stay = true;
                            mn = min(mn, d);
                        } else if (claim(u)) {
                            ++claimed;
                            // d counts the unpeeled neighbours: with none,
                            // peeling u would decrement nobody
                            pl = d > 0;
                        }
                    }
                }
                push(pl, u, rd);
                tx::find(keep, nkeep, stay, u);
                if (nkeep > tx::kBuf - 32) flush_keep();
            }
            flush_keep();
            mn = __reduce_min_sync(0xffffffffu, mn);
            if (lane == 0 && mn != INT_MAX) atomicMin(&M.ml, mn);
        }
        // drain the CTA's queue; when it runs dry, flush the gathered hub
        // decrements (the one flush that takes a degree from >= k to < k
        // pushes the vertex) and go on until nothing is left
        for (int round = 0;; ++round) {
            __syncthreads();
            uint32_t cnt = min(M.lqn[rd], (uint32_t)kLocalQ);
            if (cnt == 0) {
                if (!M.any_dec) break;
                __syncthreads();  // every thread has read any_dec
                if (threadIdx.x == 0) M.any_dec = 0;
                for (int i = threadIdx.x; i < kKcoreHubs; i += kKcoreThreads) {
                    const int32_t c = M.dec[i];
                    bool won = false;
                    if (c) {
                        M.dec[i] = 0;
                        const int32_t old = atomicSub(&deg[i], c);
                        won = old >= k && old - c < k && claim(i);
                        claimed += won;
                    }
                    push(won, i, rd);
                }
                __syncthreads();
                cnt = min(M.lqn[rd], (uint32_t)kLocalQ);
                if (cnt == 0) break;
            }
            if (round == kLocalRounds) {
                if (threadIdx.x == 0) atomicAdd(&out->rest, 1u);
                break;
            }
            const int wr = rd ^ 1;
            for (uint32_t base = 0; base < cnt; base += kKcoreThreads) {
                // rows of up to kKcoreThreads entries of the queue, end to end
                const uint32_t i = base + threadIdx.x;
                const int32_t u = i < cnt ? M.lq[rd][i] : 0;
                const uint64_t b = i < cnt ? off[u] : 0;
                const uint32_t len = i < cnt ? (uint32_t)min(off[u + 1] - b, (uint64_t)(1u << 21)) : 0;
                uint32_t end = len;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t x = __shfl_up_sync(0xffffffffu, end, o);
                    if (lane >= o) end += x;
                }
                if (lane == 31) M.warp_sum[warp] = end;
                __syncthreads();
                uint32_t total = 0;
                for (int x = 0; x < kWarps; ++x) {
                    const uint32_t y = M.warp_sum[x];
                    if (x < warp) end += y;
                    total += y;
                }
                M.tile.start[threadIdx.x] = end - len;
                M.tile.base[threadIdx.x] = b - (end - len);
                __syncthreads();
                if (total > local_edges) {  // too much for one CTA: the next step shares it among all
                    tx::find(spill, nspill, i < cnt, u);
                    if (nspill > tx::kBuf - 32) tx::flush(spill, nspill, off, QN, &out->nl, &out->nh);
                    continue;
                }
                for (uint32_t e0 = 0; e0 < total; e0 += kKcoreThreads * tx::kPerLane) {
                    uint64_t j[tx::kPerLane];
                    bool ok[tx::kPerLane];
#pragma unroll
                    for (int x = 0; x < tx::kPerLane; ++x) {
                        const uint32_t e = e0 + x * kKcoreThreads + threadIdx.x;
                        ok[x] = e < total;
                        int lo = 0;
#pragma unroll
                        for (int s = kKcoreThreads / 2; s; s >>= 1)
                            if (M.tile.start[lo + s] <= e) lo += s;
                        j[x] = M.tile.base[lo] + e;
                    }
                    peel_entries(j, ok, wr);
                }
                __syncthreads();  // the tile is rewritten
            }
            __syncthreads();
            if (threadIdx.x == 0) M.lqn[rd] = 0;
            rd = wr;
        }
        tx::flush(spill, nspill, off, QN, &out->nl, &out->nh);
        claimed = __reduce_add_sync(0xffffffffu, claimed);
        if (lane == 0 && claimed) atomicAdd(&M.claimed, claimed);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (M.claimed) atomicAdd(&out->claimed, M.claimed);
            if (M.ml != INT_MAX) atomicMin(&out->ml, M.ml);
            M.claimed = 0;
            M.ml = INT_MAX;
        }
        if (!grid_sync(gb, limit_ns)) return;
    }
    if (lead) atomicExch(&gb->err, 2);
}

// Self-test of the grid barrier: `rounds` barriers, each CTA adding 1 to
// `tally` before each; CTA `absent` (if >= 0) never arrives, so the others'
// waits run out after limit_ns and the barrier reports it.
__global__ void k_grid_sync_selftest(GridBarrier* gb, int rounds, int absent, uint64_t limit_ns,
                                     unsigned* tally, unsigned* bad) {
    if ((int)blockIdx.x == absent) return;
    for (int r = 0; r < rounds; ++r) {
        if (threadIdx.x == 0) atomicAdd(tally, 1u);
        if (!grid_sync(gb, limit_ns)) return;
        // after barrier r every CTA has added its r+1 increments
        if (threadIdx.x == 0 && __ldcg(tally) < (unsigned)(r + 1) * gridDim.x) atomicAdd(bad, 1u);
        if (!grid_sync(gb, limit_ns)) return;
    }
}

// ---- MIS -------------------------------------------------------------------------
//
// The lexicographically-first set: u is in it when no neighbour of smaller
// priority is.  Work-efficient form (Blelloch, Fineman, Shun, "Greedy
// sequential maximal independent set and matching are parallel on average",
// SPAA 2012): waits[u] counts the undecided neighbours of smaller priority; a
// vertex that is decided is queued once, and its row tells its neighbours: a
// member takes its undecided neighbours out, a vertex left out stops the
// neighbours of larger priority from waiting, and the one that waits for
// nobody any more is a member.  Every decision follows from final ones, so the
// order does not matter and the set is unique.
//
// One persistent kernel: a step expands the queue of the vertices decided in
// the step before (tx::expand); every entry is looked at once (and once more to
// count, under priorities that are not the ids).  Bound by the steps' latency
// on small graphs, by the gathers of states on large ones.  Rounds over the
// undecided vertices' whole rows, a launch and a host read each, took 0.32 ms
// at RMAT-16 and 3.1 at RMAT-22 (hashed), 4.2 at RMAT-22 under ids; this form
// 0.19, 1.9 and 1.6 ms.
//
// The kernel ends when all vertices are decided, without a look at the last
// ones' rows: a bipartite graph of 100 rows of 100 K entries takes 84 us, with
// that look 122, 4000 cliques of 64 vertices 70 and 135.  (The rounds, which
// stop at a row's first member, took 58 us for the former, and 172 against 366
// under hashed priorities, whose count looks at every entry.)  Five CTAs an SM:
// with six the count of the decided spills (RMAT-22 1.61 ms, 1.56 with five).
struct __align__(16) MisState {
    uint32_t nl, nh;  // the queues of the step that reads the record
    int32_t par;
    uint32_t done;    // vertices decided before it
};

// Priorities: a hash of the caller's id, or that id; ties by internal id.
struct MisPriority {
    uint64_t key;
    int hashed;
    const int32_t* __restrict__ int2api;  // null: the same ids
    __device__ __forceinline__ bool less(int32_t v, int32_t u) const {  // v before u
        const uint32_t a = int2api ? (uint32_t)int2api[v] : (uint32_t)v, b = int2api ? (uint32_t)int2api[u] : (uint32_t)u;
        const uint64_t pv = hashed ? pc_vertex_priority(key, a) : a, pu = hashed ? pc_vertex_priority(key, b) : b;
        return pv < pu || (pv == pu && v < u);
    }
};

// state: -1 undecided, 0 left out, 1 member.  dplus (id priorities): the
// neighbours to wait for; else every vertex is queued to have them counted.
__global__ void k_mis_init(const uint64_t* __restrict__ off, uint64_t n, const uint32_t* __restrict__ dplus,
                           int32_t* __restrict__ state, int32_t* __restrict__ waits, tx::Queues Q, MisState* S,
                           GridBarrier* gb) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *gb = GridBarrier{};
    __shared__ tx::Buffer buf[kThreads / 32];
    tx::Buffer& B = buf[threadIdx.x >> 5];
    uint32_t nb = 0;
    for (uint64_t u0 = blockIdx.x * (uint64_t)blockDim.x; u0 < n; u0 += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t u = u0 + threadIdx.x;
        if (u < n) {
            state[u] = -1;
            waits[u] = dplus ? (int32_t)dplus[u] : 0;
        }
        if (!dplus) {
            tx::find(B, nb, u < n, (int32_t)u);
            if (nb > tx::kBuf - 32) tx::flush(B, nb, off, Q, &S[0].nl, &S[0].nh);
        }
    }
    tx::flush(B, nb, off, Q, &S[0].nl, &S[0].nh);
}

__global__ void __launch_bounds__(tx::kThreads, 5)
    k_mis_persistent(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj, uint64_t n, MisPriority P,
                     int count_first, int32_t* state, int32_t* waits, tx::Queues q0, tx::Queues q1, MisState* S,
                     GridBarrier* gb, uint64_t max_steps, uint64_t limit_ns) {
    __shared__ tx::Tile s_tile[tx::kWarps];
    __shared__ tx::Buffer s_buf[tx::kWarps];
    __shared__ uint32_t s_found;
    tx::Tile& T = s_tile[threadIdx.x >> 5];
    tx::Buffer& B = s_buf[threadIdx.x >> 5];
    uint32_t nb = 0;
    if (threadIdx.x == 0) s_found = 0;
    __syncthreads();
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    const int lane = threadIdx.x & 31;
    const uint64_t first = count_first ? 1 : 0;  // step in which the vertices that wait for nobody join
    uint64_t step = 0;
    for (; step < max_steps; ++step) {
        const MisState* in = &S[step % 3];
        MisState* out = &S[(step + 1) % 3];
        const int4 r = __ldcg(reinterpret_cast<const int4*>(in));
        const uint32_t nl = (uint32_t)r.x, nh = (uint32_t)r.y;
        const int32_t par = r.z;
        const uint32_t done = (uint32_t)r.w;
        // every CTA reads the same record, so all leave at the same step; when
        // all are decided, the last ones' rows have nobody left to tell
        if (step > first && ((!nl && !nh) || done == n)) return;
        uint32_t found = 0;  // vertices the warp decided
        if (lead) {
            MisState* clr = &S[(step + 2) % 3];
            clr->nl = clr->nh = clr->done = 0;
            out->par = 1 - par;
            found = done;
        }
        const tx::Queues& Q = par ? q1 : q0;
        const tx::Queues& QN = par ? q0 : q1;
        auto flush = [&]() {
            found += nb;
            tx::flush(B, nb, off, QN, &out->nl, &out->nh);
        };
        auto room = [&]() {
            if (nb > tx::kBuf - tx::kRound) flush();
        };
        if (step < first) {
            // neighbours of smaller priority, a vote per run of lanes with the same row
            tx::expand(
                T, off, Q, nl, nh, [](int32_t u) { return u; },
                [&](const uint64_t* j, const int32_t* u, const bool* ok) {
                    int32_t v[tx::kPerLane];
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) v[k] = ok[k] ? __ldcs(adj + j[k]) : 0;
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) {
                        const unsigned m = __ballot_sync(0xffffffffu, ok[k] && P.less(v[k], u[k]));
                        if (!m) continue;
                        const unsigned run = __match_any_sync(0xffffffffu, u[k]);
                        if (lane == __ffs(run) - 1 && (m & run)) atomicAdd(&waits[u[k]], __popc(m & run));
                    }
                },
                []() {});
        } else if (step == first) {
            for (uint64_t u0 = blockIdx.x * (uint64_t)tx::kThreads; u0 < n; u0 += (uint64_t)gridDim.x * tx::kThreads) {
                const uint64_t u = u0 + threadIdx.x;
                const bool in_set = u < n && __ldcg(waits + u) == 0;
                if (in_set) state[u] = 1;
                const bool row = in_set && off[u + 1] > off[u];
                found += __popc(__ballot_sync(0xffffffffu, in_set && !row));
                tx::find(B, nb, row, (int32_t)u);
                room();
            }
        } else {
            tx::expand(
                T, off, Q, nl, nh, [&](int32_t u) { return __ldcg(state + u) ? u : ~u; },
                [&](const uint64_t* j, const int32_t* val, const bool* ok) {
                    int32_t v[tx::kPerLane];
                    bool hit[tx::kPerLane];
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) v[k] = ok[k] ? __ldcs(adj + j[k]) : 0;
                    // a state read here may be an old "undecided" from L1: a member's
                    // row settles that by compare-and-swap, and a decided
                    // vertex's count is not looked at any more
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) hit[k] = ok[k] && state[v[k]] < 0;
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) {
                        if (!hit[k]) continue;
                        if (val[k] >= 0) hit[k] = atomicCAS(&state[v[k]], -1, 0) == -1;
                        else hit[k] = P.less(~val[k], v[k]) && atomicSub(&waits[v[k]], 1) == 1;
                    }
#pragma unroll
                    for (int k = 0; k < tx::kPerLane; ++k) {
                        // a vertex with a member among the neighbours it waits for
                        // never stops waiting, so no other step decides this one
                        if (hit[k] && val[k] < 0) state[v[k]] = 1;
                        tx::find(B, nb, hit[k], v[k]);
                    }
                },
                room);
        }
        flush();
        if (lane == 0 && found) atomicAdd(&s_found, found);
        __syncthreads();
        if (threadIdx.x == 0 && s_found) {
            atomicAdd(&out->done, s_found);
            s_found = 0;
        }
        if (!grid_sync(gb, limit_ns)) return;
    }
    if (lead) atomicExch(&gb->err, 2);
}

// ---- pull sweeps: PageRank and CDLP ---------------------------------------------
//
// A sweep combines, for every row, the values its ids have in a vector.  The
// gathers bound it: at RMAT-22 a third of the 128 M hit L1 and the others move
// a 32-byte sector each from L2.  (A copy of the hubs' values in shared memory
// takes up to 58 % of them, but costs the resident warps that hide the rest's
// latency: 64 / 128 / 192 KB 9.0 / 10.3 / 10.8 ms for 20 iterations against
// 8.1 without; cache hints that keep hubs in L1 and others out: 8.1-9.0.)
//
// Rows longer than PullRows::warp_deg get a warp and than cta_deg a CTA, the
// others kPullLanes lanes.  The bounds follow the graph's size (pull_rows): a
// large sweep wants few lanes per row, a small one has lanes to spare and ends
// when its longest row does.  A CTA for every row past 256 entries spent a
// third of its time in barriers: a call at RMAT-22 took 10.9 ms, now 7.9.  Every
// reduction runs in a fixed order, so results are reproducible.
struct PullRows {
    const int32_t* __restrict__ cta;
    const int32_t* __restrict__ warp;
    uint32_t ncta, nwarp;
    uint32_t cta_deg, warp_deg;
};

// cnt[0], cnt[1]: lengths of the lists.
__global__ void k_pull_rows(const uint64_t* __restrict__ off, uint64_t n, uint32_t cta_deg, uint32_t warp_deg,
                            int32_t* __restrict__ cta, int32_t* __restrict__ warp, uint32_t* __restrict__ cnt) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t nr = (n + 31) & ~31ull;
    for (uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; u < nr; u += stride) {
        const uint64_t d = u < n ? off[u + 1] - off[u] : 0;
        warp_append(d > cta_deg, (int32_t)u, cta, &cnt[0]);
        warp_append(d > warp_deg && d <= cta_deg, (int32_t)u, warp, &cnt[1]);
    }
}

// Combines the values of the ids of adj[b, e) taken by lane gl of L lanes into
// acc, four ids per 16-byte load: the loads start at the 16-byte boundary at
// or below b and step by 4 L ids; ids outside [b, e) are not looked up.  A load may
// run up to 3 ids past e, which the 64 ids of padding after the last row keep
// inside the adjacency array.  The adjacency is read once per sweep, so its
// loads carry the streaming hint (evict first): the gathered vector keeps its
// L2 lines.
//
// A CTA's rows are long and often few, and nothing else hides the latency of a
// load and its gathers: a thread takes two vectors a step and loads the next two
// while it gathers these (20 iterations, fp32 / fp64 / CDLP in ms, one vector and
// none ahead against this: star of 1 M leaves 8.8 / 9.6 / 9.2 and 5.4 / 5.9 / 5.9,
// 100 rows of 100 K entries 1.85 / 1.78 / 1.81 and 1.16 / 1.17 / 1.12, RMAT-20
// 1.96 / 2.34 / 2.17 and 1.84 / 2.24 / 2.09; one ahead 8.2 / 6.6 / 8.5 for the
// star, two together without the next 8.5 / 6.1 / 5.6).
template <int L, class Op>
__device__ __forceinline__ void pull_row(const int32_t* __restrict__ adj, uint64_t b, uint64_t e, int gl, const Op& op,
                                         typename Op::A& acc) {
    constexpr int U = L == kThreads ? 2 : 1;     // vectors a step
    constexpr bool kAhead = L == kThreads;
    // positions are relative to the boundary; the ids at [lo, lo + len) are the row's
    const int4* p = reinterpret_cast<const int4*>(adj + (b & ~3ull));
    const uint32_t lo = (uint32_t)b & 3u, len = (uint32_t)(e - b), hi = lo + len;
    int4 v[U];
    auto load = [&](uint32_t q0) {
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = 4 * (q0 + u * L) < hi ? __ldcs(p + q0 + u * L) : make_int4(0, 0, 0, 0);
    };
    if (kAhead) load(gl);
    for (uint32_t q0 = gl; 4 * q0 < hi; q0 += U * L) {
        if (!kAhead) load(q0);
        typename Op::V x[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int32_t id[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
            for (int k = 0; k < 4; ++k) x[u][k] = 4 * (q0 + u * L) + k - lo < len ? __ldg(op.in + id[k]) : Op::none();
        }
        if (kAhead) load(q0 + U * L);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int k = 0; k < 4; ++k) op.add(acc, x[u][k]);
    }
}

template <class Op>
__global__ void __launch_bounds__(kThreads, 8)
    k_pull(const uint64_t* __restrict__ off, const int32_t* __restrict__ adj, uint64_t n, Op op, PullRows R) {
    using A = typename Op::A;
    __shared__ A s_part[kThreads / 32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (uint32_t h = blockIdx.x; h < R.ncta; h += gridDim.x) {
        const int32_t v = R.cta[h];
        A acc = Op::zero();
        pull_row<kThreads>(adj, off[v], off[v + 1], threadIdx.x, op, acc);
        for (int o = 16; o; o >>= 1) acc = Op::merge(acc, __shfl_xor_sync(0xffffffffu, acc, o));
        if (lane == 0) s_part[wib] = acc;
        __syncthreads();
        if (threadIdx.x == 0) {
            A t = Op::zero();
            for (int i = 0; i < kThreads / 32; ++i) t = Op::merge(t, s_part[i]);
            op.finish(v, off[v + 1] - off[v], t);
        }
        __syncthreads();
    }
    const uint64_t warp = (blockIdx.x * (uint64_t)kThreads + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * kThreads) >> 5;
    for (uint64_t h = warp; h < R.nwarp; h += nwarps) {
        const int32_t v = R.warp[h];
        const uint64_t b = off[v], e = off[v + 1];
        A acc = Op::zero();
        pull_row<32>(adj, b, e, lane, op, acc);
        for (int o = 16; o; o >>= 1) acc = Op::merge(acc, __shfl_xor_sync(0xffffffffu, acc, o));
        if (lane == 0) op.finish(v, e - b, acc);
    }
    // the other rows: kPullLanes lanes each, 32 / kPullLanes rows per warp at once
    constexpr int kRows = 32 / kPullLanes;
    const int g = lane / kPullLanes, gl = lane % kPullLanes;
    for (uint64_t v0 = warp * kRows; v0 < n; v0 += nwarps * kRows) {
        const uint64_t v = v0 + g;
        const uint64_t b = v < n ? off[v] : 0, e = v < n ? off[v + 1] : 0;
        const bool mine = v < n && e - b <= R.warp_deg;
        A acc = Op::zero();
        pull_row<kPullLanes>(adj, b, mine ? e : b, gl, op, acc);
        for (int o = kPullLanes / 2; o; o >>= 1) acc = Op::merge(acc, __shfl_xor_sync(0xffffffffu, acc, o));
        if (mine && gl == 0) op.finish(v, e - b, acc);
    }
}

// ---- PageRank (pull) -----------------------------------------------------------

template <class T>
__global__ void k_pr_init(const uint64_t* __restrict__ off, uint64_t n, T damping, const T* __restrict__ init,
                          T* __restrict__ contrib) {
    uint64_t u = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (u >= n) return;
    // degs[u] = d(u) / damping; x0 = degs / n (src/Graph.cpp:1563-1570)
    const T dg = (T)(off[u + 1] - off[u]) / damping;
    const T x0 = init ? init[u] : dg / (T)n;
    contrib[u] = dg > (T)0 ? x0 / dg : (T)0;
}

// One iteration: x'[v] = base + sum_{u in N(v)} contrib[u]; contrib'[v] = x'[v] / degs[v].
// T is the storage type of the vectors; the row sums, x' and the division
// run in fp64 for both instances, so the fp32 vectors carry only their own
// storage rounding (within 1e-6 relative of the FP64 recurrence at 20
// iterations; fp32 row sums over hub in-lists drift past that).  The last
// iteration writes x' (out_x), the others the contributions.
template <class T>
struct PageRankOp {
    using V = T;
    using A = double;
    const T* __restrict__ in;
    T* __restrict__ out;
    double base;
    T damping;
    bool out_x;
    static __device__ __forceinline__ A zero() { return 0.0; }
    static __device__ __forceinline__ V none() { return (V)0; }
    static __device__ __forceinline__ void add(A& a, V v) { a += (double)v; }
    static __device__ __forceinline__ A merge(A a, A b) { return a + b; }
    __device__ __forceinline__ void finish(uint64_t v, uint64_t degree, A sum) const {
        const double x = base + sum;
        const double dg = (double)((T)degree / damping);
        out[v] = out_x ? (T)x : (dg > 0.0 ? (T)(x / dg) : (T)0);
    }
};

// ---- CDLP --------------------------------------------------------------------------

// One iteration: out[v] = max label over N(v), 0 for an isolated vertex
// (src/Graph.cpp:650: labels start at 0 for every vertex).
struct CdlpOp {
    using V = int32_t;
    using A = int32_t;
    const int32_t* __restrict__ in;
    int32_t* __restrict__ out;
    static __device__ __forceinline__ A zero() { return 0; }
    static __device__ __forceinline__ V none() { return 0; }
    static __device__ __forceinline__ void add(A& a, V v) { a = max(a, v); }
    static __device__ __forceinline__ A merge(A a, A b) { return max(a, b); }
    __device__ __forceinline__ void finish(uint64_t v, uint64_t, A m) const { out[v] = m; }
};

}  // namespace fr

using namespace fr;

static unsigned grid_for(const pc_pgraph* pg, int per_sm = 8) { return (unsigned)(sm_count(pg->g->device) * per_sm); }

// CTAs of a persistent kernel: every SM's share, fewer for a small graph,
// whose barriers then have fewer arrivals; one per `work` vertices and quarter
// entries.  BFS takes 2048 (RMAT-16: 0.14 ms, 0.20 with 256), SSSP, whose steps
// wait on chains of atomics, 256 (RMAT-16: 0.37 ms, 0.41 with 2048), MIS 1024,
// k-core's larger CTAs 4096.
static pc_status persistent_grid(const pc_pgraph* pg, const void* kernel, int threads, int most_per_sm, uint64_t work,
                                 unsigned* grid, size_t smem = 0) {
    int per_sm = 0;
    PC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    if (per_sm < 1) return fail(PC_ERR_CUDA, "persistent kernel cannot be resident");
    const uint64_t all = (uint64_t)sm_count(pg->g->device) * std::min(per_sm, most_per_sm);
    *grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(all, ceil_div(pg->g->n + pg->g->m / 4, work)));
    return PC_OK;
}

static pc_status bfs_run(pc_pgraph* pg, int32_t src, int32_t* rank_host) {
    const uint64_t n = pg->g->n, m = pg->g->m;
    cudaStream_t s = pg->g->stream;
    const uint64_t hcap = tx::heavy_chunks(n, m);
    PC_TRY(scratch_reserve(pg, n * 4 * 4 + hcap * 16 + 1024));
    int32_t* dist = pg->scratch.take<int32_t>(n);
    int32_t* out = pg->scratch.take<int32_t>(n);
    tx::Queues q0{pg->scratch.take<int32_t>(n), nullptr}, q1{pg->scratch.take<int32_t>(n), nullptr};
    q0.heavy = pg->scratch.take<int2>(hcap);
    q1.heavy = pg->scratch.take<int2>(hcap);
    BfsState* S = pg->scratch.take<BfsState>(3);
    GridBarrier* gb = pg->scratch.take<GridBarrier>(1);
    if (!gb) return fail(PC_ERR_OOM, "BFS scratch plan exceeds its reservation");
    PC_CUDA(cudaMemsetAsync(gb, 0, sizeof(GridBarrier), s));
    k_bfs_init<<<grid_for(pg), kThreads, 0, s>>>(pg->off, n, m, src, dist, q0, S);
    PC_LAUNCHED();
    unsigned grid = 0;
    PC_TRY(persistent_grid(pg, (const void*)k_bfs_persistent, tx::kThreads, 6, 2048, &grid));
    uint64_t max_steps = 2 * (n + 1) + 64, limit_ns = barrier_limit_ns(), nn = n;
    const uint64_t* off = pg->off;
    const int32_t* adj = pg->adj;
    void* args[] = {(void*)&off, (void*)&adj, (void*)&nn, (void*)&src, (void*)&dist,      (void*)&q0,
                    (void*)&q1,  (void*)&S,   (void*)&gb, (void*)&max_steps, (void*)&limit_ns};
    PC_CUDA(cudaLaunchCooperativeKernel((const void*)k_bfs_persistent, dim3(grid), dim3(tx::kThreads), args, 0, s));
    PC_LAUNCHED();
    if (!api_is_internal(pg)) {
        PC_TRY(gather_to_api_i32(pg, dist, out));
        dist = out;
    }
    GridBarrier hb{};
    PC_CUDA(cudaMemcpyAsync(&hb, gb, sizeof(hb), cudaMemcpyDeviceToHost, s));
    PC_CUDA(cudaMemcpyAsync(rank_host, dist, n * 4, cudaMemcpyDeviceToHost, s));
    PC_TRY(sync(pg));
    if (hb.err == 1) return fail(PC_ERR_TIMEOUT, "BFS: a grid barrier wait ran out of time");
    if (hb.err) return fail(PC_ERR_TIMEOUT, "BFS did not converge");
    return PC_OK;
}

// Bounds of the row classes, measured with PageRank's 20 iterations on RMAT
// graphs (ms): warp_deg 32 / 64 / 128 / 256 / 512 at scale 14 (0.5 M entries)
// 0.26 / 0.22 / 0.28 / 0.35 / -, at 18 (8 M) 0.57 / 0.56 / 0.55 / 0.61 / -, at 22
// (128 M) - / - / 8.04 / 8.09 / 7.53; cta_deg 512 / 1024 / 2048 / 4096 at 16
// 0.29 / 0.29 / 0.31 / 0.31, at 20 2.39 / 2.35 / 1.91 / 2.06.
static uint32_t pull_warp_deg(uint64_t m) { return m >= (1ull << 26) ? 512 : (m >= (1ull << 22) ? 128 : 64); }
static uint32_t pull_cta_deg(uint64_t m) { return m >= (1ull << 24) ? 2048 : 1024; }

// Device bytes pull_rows() takes from the scratch arena.
static uint64_t pull_rows_bytes(uint64_t n, uint64_t m) {
    return (std::min<uint64_t>(n, m / pull_cta_deg(m)) + std::min<uint64_t>(n, m / pull_warp_deg(m)) + 2) * 4 + 1024;
}

// Lists the long rows; waits for the stream.
static pc_status pull_rows(pc_pgraph* pg, PullRows* rows) {
    const uint64_t n = pg->g->n, m = pg->g->m;
    const uint32_t cta_deg = pull_cta_deg(m), warp_deg = pull_warp_deg(m);
    cudaStream_t s = pg->g->stream;
    int32_t* cta = pg->scratch.take<int32_t>(std::min<uint64_t>(n, m / cta_deg) + 1);
    int32_t* warp = pg->scratch.take<int32_t>(std::min<uint64_t>(n, m / warp_deg) + 1);
    uint32_t* cnt = pg->scratch.take<uint32_t>(2);
    if (!cnt) return fail(PC_ERR_OOM, "scratch plan exceeds its reservation");
    PC_CUDA(cudaMemsetAsync(cnt, 0, 8, s));
    k_pull_rows<<<(unsigned)std::min<uint64_t>(grid_for(pg), ceil_div(n, kThreads)), kThreads, 0, s>>>(
        pg->off, n, cta_deg, warp_deg, cta, warp, cnt);
    PC_LAUNCHED();
    uint32_t h[2] = {0, 0};
    PC_CUDA(cudaMemcpyAsync(h, cnt, 8, cudaMemcpyDeviceToHost, s));
    PC_CUDA(cudaStreamSynchronize(s));
    *rows = PullRows{cta, warp, h[0], h[1], cta_deg, warp_deg};
    return PC_OK;
}

template <class Op>
static pc_status pull_sweep(pc_pgraph* pg, const Op& op, const PullRows& rows) {
    const uint64_t n = pg->g->n;
    // a CTA for each CTA row, a warp for each warp row, a lane group for each other one
    const uint64_t work = std::max<uint64_t>(rows.ncta, std::max<uint64_t>(ceil_div(rows.nwarp, kThreads / 32),
                                                                           ceil_div(n, kThreads / kPullLanes)));
    const uint64_t grid = std::min<uint64_t>(grid_for(pg, 16), work);
    k_pull<Op><<<(unsigned)grid, kThreads, 0, pg->g->stream>>>(pg->off, pg->adj, n, op, rows);
    PC_LAUNCHED();
    return PC_OK;
}

template <class T>
static pc_status pagerank_run(pc_pgraph* pg, T damping, int32_t iters, const T* init, T* out_host) {
    const uint64_t n = pg->g->n;
    cudaStream_t s = pg->g->stream;
    PC_TRY(scratch_reserve(pg, n * sizeof(T) * 4 + pull_rows_bytes(n, pg->g->m)));
    T* c0 = pg->scratch.take<T>(n);
    T* c1 = pg->scratch.take<T>(n);
    T* xapi = pg->scratch.take<T>(n);
    T* ini = nullptr;
    if (init) {
        ini = pg->scratch.take<T>(n);
        PC_CUDA(cudaMemcpyAsync(xapi, init, n * sizeof(T), cudaMemcpyHostToDevice, s));
        if (sizeof(T) == 4) PC_TRY(gather_to_internal_f32(pg, (const float*)xapi, (float*)ini));
        else PC_TRY(gather_to_internal_f64(pg, (const double*)xapi, (double*)ini));
    }
    k_pr_init<T><<<(unsigned)ceil_div(n, kThreads), kThreads, 0, s>>>(pg->off, n, damping, ini, c0);
    PC_LAUNCHED();
    PullRows rows;
    PC_TRY(pull_rows(pg, &rows));
    // (1 - damping) / n (src/Graph.cpp:1558), in fp64 like the row sums
    const double base = (1.0 - (double)damping) / (double)n;
    for (int32_t it = 0; it < iters; ++it) {
        PC_TRY(pull_sweep(pg, PageRankOp<T>{c0, c1, base, damping, it + 1 == iters}, rows));
        std::swap(c0, c1);
    }
    if (!api_is_internal(pg)) {
        if (sizeof(T) == 4) PC_TRY(gather_to_api_f32(pg, (const float*)c0, (float*)xapi));
        else PC_TRY(gather_to_api_f64(pg, (const double*)c0, (double*)xapi));
        c0 = xapi;
    }
    PC_CUDA(cudaMemcpyAsync(out_host, c0, n * sizeof(T), cudaMemcpyDeviceToHost, s));
    return sync(pg);
}

static pc_status mis_run(pc_pgraph* pg, bool hashed, uint64_t seed, int32_t* res_host) {
    const uint64_t n = pg->g->n, m = pg->g->m;
    cudaStream_t s = pg->g->stream;
    const int32_t* int2api = api_is_internal(pg) ? nullptr : pg->old2new.as<int32_t>();
    // under the internal ids themselves the neighbours to wait for are the
    // first dplus[u] of a row
    const bool count_first = hashed || int2api;
    if (!count_first) PC_TRY(ensure_dplus(pg));
    // a step decides a vertex once; where an adjacency that was not checked is
    // not symmetric, it may do so twice, as left out and as waiting for nobody
    const uint64_t twice = pg->g->checked ? 1 : 2, lcap = twice * n, hcap = twice * tx::heavy_chunks(n, m);
    PC_TRY(scratch_reserve(pg, n * 4 * 3 + lcap * 8 + hcap * 16 + 1024));
    int32_t* state = pg->scratch.take<int32_t>(n);
    int32_t* waits = pg->scratch.take<int32_t>(n);
    int32_t* out = pg->scratch.take<int32_t>(n);
    tx::Queues q0{pg->scratch.take<int32_t>(lcap), nullptr}, q1{pg->scratch.take<int32_t>(lcap), nullptr};
    q0.heavy = pg->scratch.take<int2>(hcap);
    q1.heavy = pg->scratch.take<int2>(hcap);
    MisState* S = pg->scratch.take<MisState>(3);
    GridBarrier* gb = pg->scratch.take<GridBarrier>(1);
    if (!gb) return fail(PC_ERR_OOM, "MIS scratch plan exceeds its reservation");
    PC_CUDA(cudaMemsetAsync(S, 0, 3 * sizeof(MisState), s));
    const unsigned nb = (unsigned)std::min<uint64_t>(grid_for(pg), ceil_div(n, kThreads));
    k_mis_init<<<nb, kThreads, 0, s>>>(pg->off, n, count_first ? nullptr : pg->dplus.as<uint32_t>(), state, waits, q0, S,
                                       gb);
    PC_LAUNCHED();
    unsigned grid = 0;
    PC_TRY(persistent_grid(pg, (const void*)k_mis_persistent, tx::kThreads, 5, 1024, &grid));
    uint64_t max_steps = 2 * n + 8, limit_ns = barrier_limit_ns(), nn = n;
    const uint64_t* off = pg->off;
    const int32_t* adj = pg->adj;
    MisPriority P{pc_graph_key(seed, PC_GEN_PRIORITY), hashed ? 1 : 0, int2api};
    int first = count_first ? 1 : 0;
    void* args[] = {(void*)&off, (void*)&adj, (void*)&nn, (void*)&P, (void*)&first, (void*)&state, (void*)&waits,
                    (void*)&q0,  (void*)&q1,  (void*)&S,  (void*)&gb, (void*)&max_steps, (void*)&limit_ns};
    PC_CUDA(cudaLaunchCooperativeKernel((const void*)k_mis_persistent, dim3(grid), dim3(tx::kThreads), args, 0, s));
    PC_LAUNCHED();
    if (!api_is_internal(pg)) {
        PC_TRY(gather_to_api_i32(pg, state, out));
        state = out;
    }
    GridBarrier hb{};
    PC_CUDA(cudaMemcpyAsync(&hb, gb, sizeof(hb), cudaMemcpyDeviceToHost, s));
    PC_CUDA(cudaMemcpyAsync(res_host, state, n * 4, cudaMemcpyDeviceToHost, s));
    PC_TRY(sync(pg));
    if (hb.err == 1) return fail(PC_ERR_TIMEOUT, "MIS: a grid barrier wait ran out of time");
    if (hb.err) return fail(PC_ERR_TIMEOUT, "MIS did not converge");
    return PC_OK;
}

static pc_status sssp_run(pc_pgraph* pg, int32_t isrc, int32_t method, int32_t delta, int32_t* dist_host) {
    const uint64_t n = pg->g->n, m = pg->g->m;
    const bool use_delta = method != PC_SSSP_BELLMAN_FORD;
    cudaStream_t s = pg->g->stream;
    const uint64_t hcap = tx::heavy_chunks(n, m);
    PC_TRY(scratch_reserve(pg, n * 4 * 8 + hcap * 16 + 1024));
    int32_t* dist = pg->scratch.take<int32_t>(n);
    int32_t* stamp = pg->scratch.take<int32_t>(n);
    int32_t* farflag = pg->scratch.take<int32_t>(n);
    tx::Queues q0{pg->scratch.take<int32_t>(n), nullptr}, q1{pg->scratch.take<int32_t>(n), nullptr};
    q0.heavy = pg->scratch.take<int2>(hcap);
    q1.heavy = pg->scratch.take<int2>(hcap);
    int32_t* far0 = pg->scratch.take<int32_t>(n);
    int32_t* far1 = pg->scratch.take<int32_t>(n);
    int32_t* out = pg->scratch.take<int32_t>(n);
    SsspState* S = pg->scratch.take<SsspState>(3);
    SsspFar* F = pg->scratch.take<SsspFar>(1);
    GridBarrier* gb = pg->scratch.take<GridBarrier>(1);
    int32_t* d_delta = pg->scratch.take<int32_t>(1);
    if (!d_delta) return fail(PC_ERR_OOM, "SSSP scratch plan exceeds its reservation");
    PC_CUDA(cudaMemsetAsync(gb, 0, sizeof(GridBarrier), s));
    const bool choose = use_delta && delta == 0;
    if (choose) {
        k_sssp_delta<<<1, 1024, 0, s>>>(pg->w, m, d_delta);
        PC_LAUNCHED();
    }
    // Bellman-Ford: one unbounded bucket
    k_sssp_init<<<grid_for(pg), kThreads, 0, s>>>(pg->off, n, isrc, use_delta ? delta : INT_MAX, d_delta, dist, stamp,
                                                  farflag, q0, S, F);
    PC_LAUNCHED();
    unsigned grid = 0;
    PC_TRY(persistent_grid(pg, (const void*)k_sssp_persistent, tx::kThreads, 5, 256, &grid));
    uint64_t max_steps = 8 * (n + 1) + 64, limit_ns = barrier_limit_ns();
    const uint64_t* off = pg->off;
    const int32_t* adj = pg->adj;
    const int32_t* w = pg->w;
    const int32_t* chosen = choose ? d_delta : nullptr;
    int32_t given = use_delta ? delta : INT_MAX;
    void* args[] = {(void*)&off, (void*)&adj,  (void*)&w,    (void*)&dist,   (void*)&stamp, (void*)&farflag,
                    (void*)&q0,  (void*)&q1,   (void*)&far0, (void*)&far1,   (void*)&chosen, (void*)&given,
                    (void*)&S,   (void*)&F,    (void*)&gb,   (void*)&max_steps, (void*)&limit_ns};
    PC_CUDA(cudaLaunchCooperativeKernel((const void*)k_sssp_persistent, dim3(grid), dim3(tx::kThreads), args, 0, s));
    PC_LAUNCHED();
    if (!api_is_internal(pg)) {
        PC_TRY(gather_to_api_i32(pg, dist, out));
        dist = out;
    }
    GridBarrier hb{};
    PC_CUDA(cudaMemcpyAsync(&hb, gb, sizeof(hb), cudaMemcpyDeviceToHost, s));
    PC_CUDA(cudaMemcpyAsync(dist_host, dist, n * 4, cudaMemcpyDeviceToHost, s));
    PC_TRY(sync(pg));
    if (hb.err == 1) return fail(PC_ERR_TIMEOUT, "SSSP: a grid barrier wait ran out of time");
    if (hb.err) return fail(PC_ERR_TIMEOUT, "SSSP did not converge");
    return PC_OK;
}

// Row entries of a CTA's local queue above which the queue goes to the next
// step's frontier (shared by every CTA): kLocalEdges, or PC_KCORE_LOCAL_EDGES
// from the environment (read once; a switch for measurements).
static uint32_t kcore_local_edges() {
    static const uint32_t v = [] {
        const char* e = getenv("PC_KCORE_LOCAL_EDGES");
        const long x = e ? atol(e) : (long)kLocalEdges;
        return (uint32_t)std::max(64L, std::min(x, 1L << 20));
    }();
    return v;
}

static pc_status kcore_run(pc_pgraph* pg, int32_t* core_host, int32_t* largest) {
    const uint64_t n = pg->g->n;
    cudaStream_t s = pg->g->stream;
    const uint64_t hcap = tx::heavy_chunks(n, pg->g->m);
    PC_TRY(scratch_reserve(pg, n * 4 * 7 + hcap * 16 + 1024));
    int32_t* deg = pg->scratch.take<int32_t>(n);
    int32_t* core = pg->scratch.take<int32_t>(n);
    int32_t* rem0 = pg->scratch.take<int32_t>(n);
    int32_t* rem1 = pg->scratch.take<int32_t>(n);
    tx::Queues q0{pg->scratch.take<int32_t>(n), nullptr}, q1{pg->scratch.take<int32_t>(n), nullptr};
    q0.heavy = pg->scratch.take<int2>(hcap);
    q1.heavy = pg->scratch.take<int2>(hcap);
    int32_t* out = pg->scratch.take<int32_t>(n);
    KState* S = pg->scratch.take<KState>(3);
    GridBarrier* gb = pg->scratch.take<GridBarrier>(1);
    int32_t* d_top = pg->scratch.take<int32_t>(1);
    if (!d_top) return fail(PC_ERR_OOM, "k-core scratch plan exceeds its reservation");
    // Levels k = 1 .. n-1, as the reference's loop (src/Graph.cpp:683, 1893):
    // at level k every remaining vertex of degree < k gets core k-1, and
    // peeling repeats until no degree crosses below k; empty levels jump to
    // the minimum degree left, as the reference does (src/Graph.cpp:1921).
    // Vertices never peeled (only in a complete graph) keep core 0.
    k_kcore_init<<<(unsigned)ceil_div(n, kThreads), kThreads, 0, s>>>(pg->off, n, deg, core, rem0, S, d_top, gb);
    PC_LAUNCHED();
    PC_CUDA(cudaFuncSetAttribute(k_kcore_persistent, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kKcoreSmem));
    unsigned grid = 0;
    PC_TRY(persistent_grid(pg, (const void*)k_kcore_persistent, kKcoreThreads, kKcorePerSm, 4096, &grid, kKcoreSmem));
    // a step scans a level or peels vertices claimed before it; each vertex
    // is claimed once, so n levels plus 2n peel steps bound the steps
    uint64_t max_steps = 3 * n + 8;
    uint64_t limit_ns = barrier_limit_ns();
    const uint64_t* off = pg->off;
    const int32_t* adj = pg->adj;
    uint64_t nn = n;
    uint32_t local_edges = kcore_local_edges();
    void* args[] = {(void*)&off, (void*)&adj, (void*)&nn, (void*)&deg, (void*)&core, (void*)&rem0, (void*)&rem1,
                    (void*)&q0,  (void*)&q1,  (void*)&S,  (void*)&gb,  (void*)&max_steps, (void*)&limit_ns,
                    (void*)&d_top, (void*)&local_edges};
    PC_CUDA(cudaLaunchCooperativeKernel((const void*)k_kcore_persistent, dim3(grid), dim3(kKcoreThreads), args, kKcoreSmem,
                                        s));
    PC_LAUNCHED();
    if (!api_is_internal(pg)) {
        PC_TRY(gather_to_api_i32(pg, core, out));
        core = out;
    }
    GridBarrier hb{};
    int32_t top = 0;
    PC_CUDA(cudaMemcpyAsync(&hb, gb, sizeof(hb), cudaMemcpyDeviceToHost, s));
    PC_CUDA(cudaMemcpyAsync(&top, d_top, 4, cudaMemcpyDeviceToHost, s));
    PC_CUDA(cudaMemcpyAsync(core_host, core, n * 4, cudaMemcpyDeviceToHost, s));
    PC_TRY(sync(pg));
    // the kernel's own status decides whether core_host holds a result
    if (hb.err == 1) return fail(PC_ERR_TIMEOUT, "k-core: a grid barrier wait ran out of time");
    if (hb.err) return fail(PC_ERR_TIMEOUT, "k-core peeling did not finish within its step bound");
    if (largest) *largest = top;
    return PC_OK;
}

static pc_status cdlp_run(pc_pgraph* pg, int32_t iterations, int32_t* labels) {
    const uint64_t n = pg->g->n;
    cudaStream_t s = pg->g->stream;
    PC_TRY(scratch_reserve(pg, n * 4 * 3 + pull_rows_bytes(n, pg->g->m)));
    int32_t* a = pg->scratch.take<int32_t>(n);
    int32_t* b = pg->scratch.take<int32_t>(n);
    int32_t* c = pg->scratch.take<int32_t>(n);
    if (!c) return fail(PC_ERR_OOM, "CDLP scratch plan exceeds its reservation");
    const bool same_ids = api_is_internal(pg);
    PC_CUDA(cudaMemcpyAsync(same_ids ? a : c, labels, n * 4, cudaMemcpyHostToDevice, s));
    if (!same_ids) PC_TRY(gather_to_internal_i32(pg, c, a));
    PullRows rows;
    PC_TRY(pull_rows(pg, &rows));
    for (int32_t it = 0; it < iterations; ++it) {
        PC_TRY(pull_sweep(pg, CdlpOp{a, b}, rows));
        std::swap(a, b);
    }
    if (same_ids) c = a;
    else PC_TRY(gather_to_api_i32(pg, a, c));
    PC_CUDA(cudaMemcpyAsync(labels, c, n * 4, cudaMemcpyDeviceToHost, s));
    return sync(pg);
}

}  // namespace pc

using namespace pc;

extern "C" {

pc_status pc_bfs(pc_pgraph* pg, int32_t src, int32_t* rank) {
    clear_error();
    if (!pg || !rank) return fail(PC_ERR_INVALID_INPUT, "null argument");
    const uint64_t n = pg->g->n;
    if (src < 0 || (uint64_t)src >= n) return fail(PC_ERR_INVALID_INPUT, "source vertex out of range");
    PC_TRY(use_device(pg->g));
    return with_room(pg, [&] { return bfs_run(pg, to_internal_id(pg, src), rank); });
}

pc_status pc_sssp(pc_pgraph* pg, int32_t src, int32_t* dist_host) {
    return pc_sssp_ex(pg, src, PC_SSSP_AUTO, 0, dist_host);
}

pc_status pc_sssp_ex(pc_pgraph* pg, int32_t src, int32_t method, int32_t delta, int32_t* dist_host) {
    clear_error();
    if (!pg || !dist_host) return fail(PC_ERR_INVALID_INPUT, "null argument");
    const uint64_t n = pg->g->n;
    if (!pg->w) return fail(PC_ERR_INVALID_INPUT, "SSSP needs a weighted graph");
    if (src < 0 || (uint64_t)src >= n) return fail(PC_ERR_INVALID_INPUT, "source vertex out of range");
    if (method != PC_SSSP_AUTO && method != PC_SSSP_BELLMAN_FORD && method != PC_SSSP_DELTA_STEPPING)
        return fail(PC_ERR_INVALID_INPUT, "unknown SSSP method");
    if (delta < 0) return fail(PC_ERR_INVALID_INPUT, "delta must be >= 0 (0: chosen from the graph)");
    PC_TRY(use_device(pg->g));
    return with_room(pg, [&] { return sssp_run(pg, to_internal_id(pg, src), method, delta, dist_host); });
}

pc_status pc_pagerank(pc_pgraph* pg, float damping, int32_t iterations, const float* init, float* out) {
    clear_error();
    if (!pg || !out) return fail(PC_ERR_INVALID_INPUT, "null argument");
    if (iterations <= 0) return fail(PC_ERR_INVALID_INPUT, "iterations must be positive");
    if (!(damping > 0.f && damping <= 1.f)) return fail(PC_ERR_INVALID_INPUT, "damping must be in (0, 1]");
    PC_TRY(use_device(pg->g));
    return with_room(pg, [&] { return pagerank_run<float>(pg, damping, iterations, init, out); });
}

pc_status pc_pagerank_f64(pc_pgraph* pg, double damping, int32_t iterations, const double* init, double* out) {
    clear_error();
    if (!pg || !out) return fail(PC_ERR_INVALID_INPUT, "null argument");
    if (iterations <= 0) return fail(PC_ERR_INVALID_INPUT, "iterations must be positive");
    if (!(damping > 0.0 && damping <= 1.0)) return fail(PC_ERR_INVALID_INPUT, "damping must be in (0, 1]");
    PC_TRY(use_device(pg->g));
    return with_room(pg, [&] { return pagerank_run<double>(pg, damping, iterations, init, out); });
}

pc_status pc_selftest_grid_barrier(int32_t device, int32_t rounds, int32_t absent_cta, uint32_t limit_ms,
                                   uint32_t* mismatches) {
    clear_error();
    if (rounds < 0 || !mismatches || limit_ms == 0) return fail(PC_ERR_INVALID_INPUT, "bad argument");
    PC_TRY(pc_set_device(device));
    int per_sm = 0;
    PC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_grid_sync_selftest, kThreads, 0));
    if (per_sm < 1) return fail(PC_ERR_CUDA, "self-test kernel cannot be resident");
    const int grid = sm_count(device) * std::min(per_sm, 2);
    if (absent_cta >= grid) return fail(PC_ERR_INVALID_INPUT, "absent_cta is outside the grid");
    cudaStream_t s = nullptr;
    PC_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    DevBuf buf;
    pc_status st = buf.alloc(sizeof(GridBarrier) + 16, "self-test state");
    if (st != PC_OK) {
        cudaStreamDestroy(s);
        return st;
    }
    GridBarrier* gb = buf.as<GridBarrier>();
    unsigned* tally = reinterpret_cast<unsigned*>(gb + 1);
    unsigned* bad = tally + 1;
    uint64_t limit_ns = (uint64_t)limit_ms * 1000000ull;
    void* args[] = {(void*)&gb, (void*)&rounds, (void*)&absent_cta, (void*)&limit_ns, (void*)&tally, (void*)&bad};
    GridBarrier hb{};
    unsigned hbad = 0;
    cudaError_t e = cudaMemsetAsync(buf.p, 0, sizeof(GridBarrier) + 16, s);
    if (e == cudaSuccess)
        e = cudaLaunchCooperativeKernel((const void*)k_grid_sync_selftest, dim3(grid), dim3(kThreads), args, 0, s);
    count_launch();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&hb, gb, sizeof(hb), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(&hbad, bad, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaStreamDestroy(s);
    if (e != cudaSuccess) return cuda_fail(e, "grid barrier self-test", __FILE__, __LINE__);
    *mismatches = hbad;
    if (hb.err) return fail(PC_ERR_TIMEOUT, "grid barrier: a wait ran out of time");
    return PC_OK;
}

pc_status pc_kcore(pc_pgraph* pg, int32_t* core_host, int32_t* largest) {
    clear_error();
    if (!pg || !core_host) return fail(PC_ERR_INVALID_INPUT, "null argument");
    PC_TRY(use_device(pg->g));
    if (pg->g->n == 0) {
        if (largest) *largest = 0;
        return PC_OK;
    }
    return with_room(pg, [&] { return kcore_run(pg, core_host, largest); });
}

pc_status pc_mis(pc_pgraph* pg, int32_t* res) {
    clear_error();
    if (!pg || !res) return fail(PC_ERR_INVALID_INPUT, "null argument");
    PC_TRY(use_device(pg->g));
    if (pg->g->n == 0) return PC_OK;
    return with_room(pg, [&] { return mis_run(pg, false, 0, res); });
}

pc_status pc_mis_hashed(pc_pgraph* pg, uint64_t seed, int32_t* res) {
    clear_error();
    if (!pg || !res) return fail(PC_ERR_INVALID_INPUT, "null argument");
    PC_TRY(use_device(pg->g));
    if (pg->g->n == 0) return PC_OK;
    return with_room(pg, [&] { return mis_run(pg, true, seed, res); });
}

pc_status pc_cdlp(pc_pgraph* pg, int32_t iterations, int32_t* labels) {
    clear_error();
    if (!pg || !labels) return fail(PC_ERR_INVALID_INPUT, "null argument");
    if (iterations < 0) return fail(PC_ERR_INVALID_INPUT, "iterations must be non-negative");
    PC_TRY(use_device(pg->g));
    const uint64_t n = pg->g->n;
    if (n == 0 || iterations == 0) return PC_OK;
    return with_room(pg, [&] { return cdlp_run(pg, iterations, labels); });
}

}  // extern "C"
