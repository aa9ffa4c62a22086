// Grid-wide barrier of a cooperative launch, shared by the persistent
// whole-shot kernels.
#pragma once

#include "tc_util.cuh"

namespace geo {

// Arrival counter read with acquire semantics at GPU scope.
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// One arrival per block on a counter that only grows (barrier k completes at
// k*gridDim.x arrivals).  grid_arrive, by one thread after a __syncthreads,
// publishes the block's writes (release, cumulative over the block's barrier);
// grid_wait, by one thread, waits for the target (acquire), 2 s at most, and
// sets the error word when it gives up, after which every other block's next
// wait runs out too.  Values other blocks wrote before the barrier are read
// through L2 (__ldcg) or by TMA: L1 is not coherent with them.
// A release reduction instead of a fence and an atomic, and no fence after
// the acquire: a step of a 101x121 2D shot 4.0 -> 3.6 us, of 401x401 6.0 -> 5.6.
__device__ __forceinline__ void grid_arrive(unsigned *bar) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}
__device__ __forceinline__ bool grid_wait(const unsigned *bar, unsigned target, int *err) {
    if (ld_acquire_u32(bar) >= target) return true;
    const uint64_t t0 = tc::gtimer();
    while (ld_acquire_u32(bar) < target)
        if (tc::gtimer() - t0 > 2000000000ull) {
            atomicExch(err, 1);
            return false;
        }
    return true;
}
// Both, for the whole block.
__device__ __forceinline__ bool grid_barrier(unsigned *bar, unsigned target, int *err) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        grid_arrive(bar);
        s_ok = grid_wait(bar, target, err);
    }
    __syncthreads();
    return s_ok != 0;
}

}  // namespace geo
