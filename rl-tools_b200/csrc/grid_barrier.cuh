// Grid-wide barrier of the cooperative kernels: arrivals counted in a device word, every wait with a limit. The launches are cooperative, so all CTAs are
// resident together whatever else the device runs; a wait that runs into its limit all the same (about a second) ends its launch and not the process:
//   - it sets the slot's abort word, which every other wait of the launch looks at, and the device's status word in host memory, which makes the next
//     call that needs a barrier return B200RL_ERR_DEVICE_FLAG until b200rl_device_error_clear;
//   - every CTA still leaves through grid_barrier_leave, so that the last one hands the slot on clean.
#pragma once
#include "common.cuh"

namespace b200rl {

constexpr unsigned GRID_BARRIER_SPIN_LIMIT = 1000000u;                    // polls of the barrier word (an L2 round trip each): about a second

struct GridBarrier {
    unsigned* words;                                                      // arrivals, exits, abort, unused: zeros between launches
    unsigned* status;                                                     // the device's status word, host memory
};
// `count` consecutive barriers for a launch on this stream (grid_barrier.cu)
int grid_barriers(int count, cudaStream_t stream, GridBarrier* out);
// the current device's status word: 0, or 1 once a wait has run into its limit
int grid_barrier_status(unsigned* status);
int grid_barrier_clear();

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p){
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// by one thread, after a CTA-wide barrier (the CTA's writes are then ordered before the arrival) ...
__device__ __forceinline__ void grid_barrier_arrive(const GridBarrier& bar){
    __threadfence();
    atomicAdd(bar.words, 1u);
}
// ... and by the same thread, before a CTA-wide barrier. False: the wait ran into its limit (or another CTA's did).
__device__ __forceinline__ bool grid_barrier_wait(const GridBarrier& bar, unsigned target){
    unsigned spins = 0;
    while(ld_acquire_u32(bar.words) < target){
        spins++;
        const bool expired = spins > GRID_BARRIER_SPIN_LIMIT;
        if(expired || ((spins & 63u) == 0u && ld_acquire_u32(bar.words + 2) != 0u)){
            if(expired){ atomicExch(bar.words + 2, 1u); *reinterpret_cast<volatile unsigned*>(bar.status) = 1u; }
            return false;
        }
    }
    return true;
}
// by one thread of every CTA, after its last barrier or a wait that returned false: the last of the `ctas` CTAs clears the slot for its next launch
__device__ __forceinline__ void grid_barrier_leave(const GridBarrier& bar, unsigned ctas){
    const unsigned old = atomicAdd(bar.words + 1, 1u);
    if(old == ctas - 1){ bar.words[0] = 0u; bar.words[1] = 0u; bar.words[2] = 0u; __threadfence(); }
}

}  // namespace b200rl
