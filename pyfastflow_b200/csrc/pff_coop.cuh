// Barrier over the blocks of a cooperative launch.
#pragma once
#include <cuda_runtime.h>
#include "pff_internal.h"

namespace pff {

__device__ __forceinline__ int vload(const int *p) { return *(const volatile int *)p; }

// The launch is cooperative, so every block is resident; a wait that has not ended after
// about two seconds gives up.  ctr counts arrivals from zero over the whole launch.  A block
// gives up by setting BAR_HALT in the counter while arrivals are still missing (compare and
// swap); every block that sees the bit, now or at a later barrier, gives up too.  So
// no block passes a barrier that another one gave up, and after the last barrier
// either all blocks succeeded or none did: any block's outcome is the launch's, and the
// bit stays in the counter.
// About 1.3 us over 148 blocks (one atomic and one polled load through L2); one block only
// synchronises its threads.
constexpr int BAR_HALT = 1 << 30;

struct GridBar {
    int *ctr;
    unsigned limit_ns;
    int target;
    __device__ __forceinline__ GridBar(int *counter, const BarWait &w) : ctr(counter), limit_ns(w.limit_us * 1000u), target(w.absent) {}
    __device__ __forceinline__ bool sync(int *dead)
    {
        __syncthreads();
        if (gridDim.x > 1) {
            target += gridDim.x;
            if (threadIdx.x == 0) {
                __threadfence();
                atomicAdd(ctr, 1);
                unsigned long long t0;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
                int spin = 0, seen;
                for (;;) {
                    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(ctr) : "memory");
                    if (seen >= target) break;  // all arrived, or BAR_HALT
                    if ((++spin & 15) == 0) {
                        unsigned long long t;
                        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                        if (t - t0 > limit_ns) {
                            const int was = atomicCAS(ctr, seen, seen | BAR_HALT);
                            if (was == seen) seen |= BAR_HALT;
                            else if (was < target) continue;  // an arrival in between: look again
                            else seen = was;
                            break;
                        }
                    }
                }
                __threadfence();
                if (seen & BAR_HALT) *dead = 1;
            }
            __syncthreads();
        }
        return *dead == 0;
    }
};

}  // namespace pff
