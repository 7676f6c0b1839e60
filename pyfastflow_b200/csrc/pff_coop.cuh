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
constexpr int BAR_POLLS = 32;  // about 20 us

__device__ __forceinline__ int bar_poll(const int *ctr)
{
    int seen;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(ctr) : "memory");
    return seen;
}

// The rest of a long wait for *ctr to reach target, at most limit_us; the counter's value.
static __device__ __noinline__ int bar_long_wait(int *ctr, int target, unsigned limit_us)
{
    const long long t0 = clock64();
    for (;;) {
        const int seen = bar_poll(ctr);
        if (seen >= target) return seen;
        // cycles at 1.965 GHz: a little longer at lower clocks.  The swap fails if a block has
        // arrived meanwhile: then look again
        if (clock64() - t0 > 1965LL * limit_us && atomicCAS(ctr, seen, seen | BAR_HALT) == seen) return seen | BAR_HALT;
    }
}

struct GridBar {
    int *ctr;
    const BarWait &wait;
    int target;
    __device__ __forceinline__ GridBar(int *counter, const BarWait &w) : ctr(counter), wait(w), target(w.absent) {}
    __device__ __forceinline__ bool sync(int *dead)
    {
        __syncthreads();
        if (gridDim.x > 1) {
            target += gridDim.x;
            if (threadIdx.x == 0) {
                __threadfence();
                atomicAdd(ctr, 1);
                int seen = bar_poll(ctr);
                for (int spin = 0; seen < target && spin < BAR_POLLS; ++spin) seen = bar_poll(ctr);
                if (seen < target) seen = bar_long_wait(ctr, target, wait.limit_us);
                if (seen & BAR_HALT) *dead = 1;
                __threadfence();
            }
            __syncthreads();
        }
        return *dead == 0;
    }
};

}  // namespace pff
