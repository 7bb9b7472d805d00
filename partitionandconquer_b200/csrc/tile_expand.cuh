// Edge-balanced expansion of a frontier by the warps of a persistent kernel.
//
// A frontier is a queue of rows of up to kLightRow entries and a queue of
// chunks (row, run of kHeavyRun entries) of the longer ones.  A warp takes 32
// light rows, lays them end to end (a warp scan of the lengths) and its lanes
// take the entries of that sequence in order, kPerLane each at a time; or it
// takes one chunk.  Every lane has an edge whatever the rows' lengths are,
// neighbouring lanes read neighbouring entries, and kPerLane loads of each kind
// are in flight together.  A warp per row, in contrast, waits through each
// row's chain of dependent loads (queue, offsets, ids, values) with one load in
// flight per lane: SSSP's relaxation at RMAT-22 ran at 13 % issue with 105
// cycles of L2 waiting per instruction, 5.6 ms in all.  Warps, not CTAs, take
// the tiles: CTA tiles of 256 rows lost most of it to barriers.
//
// Vertices found go to a buffer of the warp in shared memory that it empties
// into the next queues, where the rows' lengths decide the queue.
#pragma once
#include "pc_internal.cuh"

namespace pc {
namespace tx {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kPerLane = 4;             // edges per lane and round
constexpr uint32_t kRound = 32 * kPerLane;
constexpr uint32_t kLightRow = 256;     // longer rows are queued in chunks
constexpr uint32_t kHeavyRun = 256;     // entries per chunk: a hub alone in a frontier still fills many warps
constexpr uint32_t kBuf = 256;          // room of a buffer
static_assert(kBuf >= 2 * kRound, "a round may find kRound vertices");

// Chunks a graph's heavy queue can hold: every heavy row once.
inline uint64_t heavy_chunks(uint64_t n, uint64_t m) {
    const uint64_t rows = m / kLightRow < n ? m / kLightRow : n;
    return m / kHeavyRun + rows + 1;
}

struct Queues {
    int32_t* light;  // rows
    int2* heavy;     // (row, chunk)
};

// Per warp.
struct Buffer {
    int32_t v[kBuf];
};
struct Tile {
    uint64_t base[32];   // CSR entry of edge 0 of the sequence, were it in that row
    uint32_t start[32];  // first edge of each row in the sequence
    int32_t val[32];     // the caller's value of the row
};

// Adds v to the buffer of *n entries (a register, the same in all lanes) for
// every lane with pred set; all lanes call it.
__device__ __forceinline__ void find(Buffer& B, uint32_t& n, bool pred, int32_t v) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (pred) B.v[n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = v;
    n += __popc(m);
}

// Appends v[0 .. k) of each lane to the queues by their rows' lengths; all 32
// lanes call it (k may differ).  Returns the lane's row entries.  The lengths
// are loaded together and each queue takes one atomic: appending 32 at a
// time, a full buffer waited through eight chains of load and atomics.
template <int kMost>
__device__ __forceinline__ uint64_t enqueue(const int32_t* v, int k, const uint64_t* __restrict__ off, const Queues& Q,
                                            uint32_t* nlight, uint32_t* nheavy) {
    const int lane = threadIdx.x & 31;
    uint64_t entries = 0;
    uint32_t chunks[kMost];  // of a heavy row, 0 of a light one
    uint32_t nl = 0, nh = 0;
#pragma unroll
    for (int i = 0; i < kMost; ++i) {
        const uint64_t deg = i < k ? off[v[i] + 1] - off[v[i]] : 0;
        entries += deg;
        chunks[i] = deg > kLightRow ? (uint32_t)((deg + kHeavyRun - 1) / kHeavyRun) : 0u;
        nl += i < k && !chunks[i];
        nh += chunks[i];
    }
    uint32_t lend = nl, hend = nh;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, lend, o), y = __shfl_up_sync(0xffffffffu, hend, o);
        if (lane >= o) {
            lend += x;
            hend += y;
        }
    }
    uint32_t lat = 0, hat = 0;
    if (lane == 31 && lend) lat = atomicAdd(nlight, lend);
    if (lane == 31 && hend) hat = atomicAdd(nheavy, hend);
    lat = __shfl_sync(0xffffffffu, lat, 31) + lend - nl;
    hat = __shfl_sync(0xffffffffu, hat, 31) + hend - nh;
#pragma unroll
    for (int i = 0; i < kMost; ++i) {
        if (i < k && !chunks[i]) Q.light[lat++] = v[i];
        for (unsigned h = __ballot_sync(0xffffffffu, chunks[i] != 0); h; h &= h - 1) {
            // the warp writes a row's chunks together
            const int src = __ffs(h) - 1;
            const uint32_t cs = __shfl_sync(0xffffffffu, chunks[i], src), as = __shfl_sync(0xffffffffu, hat, src);
            const int32_t vs = __shfl_sync(0xffffffffu, i < k ? v[i] : 0, src);
            for (uint32_t c = lane; c < cs; c += 32) Q.heavy[as + c] = make_int2(vs, (int32_t)c);
        }
        hat += chunks[i];
    }
    return entries;
}

// Empties a buffer into the next queues; returns the row entries of this
// lane's vertices.
__device__ __forceinline__ uint64_t flush(Buffer& B, uint32_t& n, const uint64_t* __restrict__ off, const Queues& Q,
                                          uint32_t* nlight, uint32_t* nheavy) {
    constexpr int kMost = kBuf / 32;
    const uint32_t lane = threadIdx.x & 31;
    if (n == 0) return 0;
    __syncwarp();
    int32_t v[kMost];
#pragma unroll
    for (int i = 0; i < kMost; ++i) v[i] = lane + 32 * i < n ? B.v[lane + 32 * i] : 0;
    const int k = n > lane ? (int)((n - lane + 31) / 32) : 0;
    const uint64_t entries = enqueue<kMost>(v, k, off, Q, nlight, nheavy);
    __syncwarp();
    n = 0;
    return entries;
}

// Expands a frontier of nl light rows and nh chunks.  value(u) is taken once per row and chunk; visit(j, val,
// ok) handles kPerLane CSR entries j of rows with those values, the lanes of a
// warp together; after each round done() may empty buffers.
template <class Value, class Visit, class Done>
__device__ __forceinline__ void expand(Tile& T, const uint64_t* __restrict__ off, const Queues& in, uint32_t nl,
                                           uint32_t nh, Value&& value, Visit&& visit, Done&& done) {
    const int lane = threadIdx.x & 31;
    const uint32_t wpb = blockDim.x >> 5, gw = blockIdx.x * wpb + (threadIdx.x >> 5), nw = gridDim.x * wpb;
    uint64_t j[kPerLane];
    int32_t val[kPerLane];
    bool ok[kPerLane];
    for (uint32_t i = gw; i < nh; i += nw) {  // the longest rows first
        const int2 h = __ldcg(in.heavy + i);
        const uint64_t b = off[h.x] + (uint64_t)h.y * kHeavyRun;
        const uint32_t len = (uint32_t)min((uint64_t)kHeavyRun, off[h.x + 1] - b);
        const int32_t x = value(h.x);
        for (uint32_t e0 = lane; e0 < ((len + 31) & ~31u); e0 += kRound) {
#pragma unroll
            for (int k = 0; k < kPerLane; ++k) {
                ok[k] = e0 + 32 * k < len;
                j[k] = b + e0 + 32 * k;
                val[k] = x;
            }
            visit(j, val, ok);
            done();
        }
    }
    // Light rows, from the other end: the warps without a chunk begin.  A short
    // queue is spread over all warps (22 rows of up to 256 entries in one warp's
    // hands held a level up for 80 us), and a tile's rows are a tile count
    // apart: neighbours in a queue tend to have rows of the same length, above
    // all under degree-ordered ids.
    const uint32_t rows = min(32u, (nl + nw - 1) / nw);
    const uint32_t tiles = rows ? (nl + rows - 1) / rows : 0u;
    for (uint32_t t = nw - 1 - gw; t < tiles; t += nw) {
        const uint32_t i = t + lane * tiles;
        uint32_t len = 0;
        uint64_t b = 0;
        int32_t x = 0;
        if (lane < rows && i < nl) {
            const int32_t u = __ldcg(in.light + i);
            b = off[u];
            len = (uint32_t)(off[u + 1] - b);
            x = value(u);
        }
        uint32_t end = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
            if (lane >= o) end += y;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, end, 31);
        __syncwarp();
        T.start[lane] = end - len;
        T.base[lane] = b - (end - len);
        T.val[lane] = x;
        __syncwarp();
        for (uint32_t e0 = lane; e0 < ((total + 31) & ~31u); e0 += kRound) {
#pragma unroll
            for (int k = 0; k < kPerLane; ++k) {
                const uint32_t e = e0 + 32 * k;
                ok[k] = e < total;
                // last row with start <= e: an empty row shares its start with the next one
                int lo = 0;
#pragma unroll
                for (int step = 16; step; step >>= 1)
                    if (T.start[lo + step] <= e) lo += step;
                j[k] = T.base[lo] + e;
                val[k] = T.val[lo];
            }
            visit(j, val, ok);
            done();
        }
    }
}

}  // namespace tx
}  // namespace pc
