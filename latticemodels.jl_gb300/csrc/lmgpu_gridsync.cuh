// Barrier over all CTAs of a cooperative launch.
#pragma once
#include <cuda_runtime.h>

namespace lmgpu {

constexpr int kGridPolls = 1 << 21;  // bound of a barrier wait (about a second)

// Every CTA adds 1 to the counter and waits until it has reached `target` (the launch's CTAs times the
// barriers so far); what a CTA wrote before is visible to all after.  False for every thread of a CTA
// whose wait gave up: it leaves the kernel, and so do the others, whose counter cannot fill up.
// In two halves, with work between them that the other CTAs do not wait for.
__device__ __forceinline__ void grid_arrive(unsigned* ctr) {
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    }
}
__device__ __forceinline__ bool grid_wait(unsigned* ctr, unsigned target) {
    __shared__ int ok;
    if (threadIdx.x == 0) {
        int good = 1, it = 0;
        unsigned seen;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(ctr) : "memory");
            if (++it > kGridPolls) {
                good = 0;
                break;
            }
        } while ((int)(seen - target) < 0);
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// Called once by every CTA after its last barrier: the last one zeroes the counter for the next launch.
__device__ __forceinline__ void grid_leave(unsigned* ctr) {
    if (threadIdx.x == 0 && atomicAdd(ctr + 1, 1u) == gridDim.x - 1) {
        ctr[1] = 0;
        __threadfence();
        ctr[0] = 0;
    }
}

}  // namespace lmgpu
