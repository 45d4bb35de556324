// The limit of a wait inside a kernel: two seconds of polling.  What lies between
// two polls counts for MAX_STEP at most, so that the time that the process was off
// the GPU (a debugger, another process' turn) does not end a healthy wait.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define MO_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define MO_HOST_DEVICE inline
#endif

namespace mo {

struct WaitLimit {
    static constexpr uint32_t LIMIT = 2000000000u, MAX_STEP = 10000000u;  // ns
    uint32_t last, spent = 0;

    MO_HOST_DEVICE explicit WaitLimit(uint32_t now) : last(now) {}
    // now: nanoseconds of a clock, modulo 2^32
    MO_HOST_DEVICE bool over(uint32_t now) {
        const uint32_t step = now - last;
        last = now;
        spent += step < MAX_STEP ? step : MAX_STEP;
        return spent > LIMIT;
    }
};

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t wait_clock() {
    uint32_t t;
    asm volatile("mov.u32 %0, %globaltimer_lo;" : "=r"(t));
    return t;
}
#endif

}  // namespace mo
