// How long a polling thread has waited, for the bounded waits of the persistent
// kernels.
//
// A waiting thread reads the time about once a microsecond.  When another
// program's context has the GPU, all threads of this one stand still while the
// clock goes on.  A longer gap between two readings therefore says nothing about
// the threads that are waited for, and counts as kWaitGapNs at most.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define PC_HD __host__ __device__ __forceinline__
#else
#define PC_HD inline
#endif

namespace pc {

constexpr uint64_t kWaitGapNs = 100000;

struct WaitClock {
    uint64_t last, waited;
    PC_HD explicit WaitClock(uint64_t now) : last(now), waited(0) {}
    // Takes a reading; whether the waiting is above the limit.
    PC_HD bool over(uint64_t now, uint64_t limit_ns) {
        const uint64_t gap = now - last;
        last = now;
        waited += gap < kWaitGapNs ? gap : kWaitGapNs;
        return waited > limit_ns;
    }
};

}  // namespace pc
