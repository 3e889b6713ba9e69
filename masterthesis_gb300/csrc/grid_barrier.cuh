// The barrier between the steps of a one-launch time loop (star7_loop.cuh).
#pragma once

#include "tma.cuh"
#include "../../include/scafes_gb300.h"

namespace scafes {

// Ends a step for the whole grid: returns false (status set) when the other
// CTAs did not arrive in time.  The release of thread 0 after the block
// barrier publishes the block's stores; its acquire makes the others' stores
// visible to the block's loads after the second block barrier.
__device__ __forceinline__ bool grid_barrier(unsigned* arrivals, unsigned target, int* status,
                                             uint64_t limit_ns = kWaitLimitNs) {
    bool ok = true;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrivals) : "memory");
        unsigned v;
        uint64_t t0 = 0;
        for (unsigned polls = 0;; ++polls) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(arrivals) : "memory");
            if ((int)(v - target) >= 0) break;
            if ((polls & 255u) == 255u) {
                const uint64_t t = global_timer_ns();
                if (t0 == 0) t0 = t;
                if (t - t0 > limit_ns) {
                    ok = false;
                    atomicExch(status, SCAFES_ERR_TIMEOUT);
                    break;
                }
            }
        }
    }
    return __syncthreads_and(ok);
}

}  // namespace scafes
