// Grid-wide barrier for persistent kernels started with a cooperative launch
// (every CTA of the grid is resident, so every CTA can reach the barrier).
//
// Every wait is bounded by a wall-clock limit read from %globaltimer: a CTA
// that waits longer, or that sees another CTA's error, records the error and
// the barrier returns false, so the kernel can return and the host can read
// the status instead of the GPU spinning for ever.
#pragma once
#include <cstdint>

namespace pc {

struct GridBarrier {
    unsigned long long arrived;  // CTAs arrived so far, over all barriers
    int err;                     // 1: a wait ran out of time; 2: a step bound was hit
    int pad;
};

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// All threads of every CTA call it.  Writes made before it (plain stores and
// atomics) are visible to every CTA after it, to loads that bypass L1
// (__ldcg) or to atomics.
__device__ __forceinline__ bool grid_sync(GridBarrier* gb, uint64_t limit_ns) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        // The counter only grows: the arrival that this barrier waits for is
        // the next multiple of the grid's size, so nothing is reset and the
        // waiting CTAs poll the counter itself (one round trip less than a
        // generation word that the last CTA bumps).
        __threadfence();
        const unsigned long long mine = atomicAdd(&gb->arrived, 1ull);
        const unsigned long long all = (mine / gridDim.x + 1) * gridDim.x;
        if (mine + 1 != all) {
            const uint64_t t0 = global_ns();
            while (ld_acquire_u64(&gb->arrived) < all) {
                if (*(volatile int*)&gb->err) { ok = 0; break; }
                if (global_ns() - t0 > limit_ns) {
                    atomicExch(&gb->err, 1);
                    ok = 0;
                    break;
                }
                __nanosleep(32);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

}  // namespace pc
