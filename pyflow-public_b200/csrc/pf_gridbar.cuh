// pf_gridbar.cuh -- a barrier over the blocks of one cooperative launch.
#pragma once
#include <cuda_runtime.h>

namespace pf {

constexpr int kGridBarWords = 2;  // arrivals, failure; zero before the launch

// All blocks of the grid meet for the round-th time (1, 2, ...); what a block
// wrote before grid_arrive is visible to all after grid_wait, also to plain
// loads (release on the arriving, acquire on the waiting side, each extended
// to the block by its barriers).  One add and one polled word: arrivals only
// ever grow, so no block waits for a reset.  grid_wait is false in every
// thread, with word 1 set, when a wait gave up (seconds).
__device__ __forceinline__ void grid_arrive(unsigned* bar) {
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
}

__device__ __forceinline__ bool grid_wait(unsigned* bar, unsigned round) {
    __shared__ int meet_ok;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        const unsigned want = round * gridDim.x;
        int ok = 1, it = 0;
        unsigned got;
        while (true) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(bar) : "memory");
            if ((int)(got - want) >= 0) break;
            if (++it > (1 << 23) || ((volatile unsigned*)bar)[1]) { ok = 0; break; }
        }
        if (!ok) atomicExch(bar + 1, 1u);
        meet_ok = ok;
    }
    __syncthreads();
    return meet_ok != 0;
}

__device__ __forceinline__ bool grid_meet(unsigned* bar, unsigned round) {
    grid_arrive(bar);
    return grid_wait(bar, round);
}

}  // namespace pf
