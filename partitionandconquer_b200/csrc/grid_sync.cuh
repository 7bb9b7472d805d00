// Grid-wide barrier for persistent kernels started with a cooperative launch
// (every CTA of the grid is resident, so every CTA can reach the barrier).
//
// Every wait is bounded by a limit on the time from %globaltimer (less the time
// in which another program had the GPU, see WaitClock): a CTA that waits longer,
// or that sees another CTA's error, records the error and the barrier returns
// false, so the kernel can return and the host can read the status instead of
// the GPU spinning for ever.
#pragma once
#include <cstdint>

#include "wait_clock.h"

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
// atomics) are visible to every CTA after it, plain loads included: thread 0's
// fence and arrival release its CTA's writes (ordered before them by the CTA
// barrier), its acquiring read of the counter and the fence after it take the
// others' in and drop what L1 holds, and the second CTA barrier passes that on.
// During a step a plain load may still return what L1 took in earlier in it.
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
            WaitClock clock(global_ns());
            while (ld_acquire_u64(&gb->arrived) < all) {
                if (*(volatile int*)&gb->err) { ok = 0; break; }
                if (clock.over(global_ns(), limit_ns)) {
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
