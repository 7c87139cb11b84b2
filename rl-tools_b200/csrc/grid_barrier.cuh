// Grid-wide barrier of the cooperative kernels: arrivals counted in a device word, every wait with a limit. A launch that runs into the limit sets
// a sticky status word (b200rl_cooperative_pass_status) and all of its CTAs return; the launches are cooperative, so all CTAs are resident together
// whatever else the device runs.
#pragma once
#include "common.cuh"

namespace b200rl {

constexpr unsigned GRID_BARRIER_SPIN_LIMIT = 1000000u;                    // polls of the barrier word (an L2 round trip each): about a second

// Four words per slot: arrivals, exits, status (sticky), unused. Slots are handed out round-robin per launch (a captured launch keeps the slot it
// got at capture time); two launches may share a slot as long as they never run at the same time, see mlp_coop.cu.
int grid_barrier_slots(int count, unsigned** out);                        // `count` consecutive slots of 4 words

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p){
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// by one thread, after a CTA-wide barrier (the CTA's writes are then ordered before the arrival) ...
__device__ __forceinline__ void grid_barrier_arrive(unsigned* bar){
    __threadfence();
    atomicAdd(bar, 1u);
}
// ... and by the same thread, before a CTA-wide barrier. False: the wait ran into its limit (or another CTA's did).
__device__ __forceinline__ bool grid_barrier_wait(unsigned* bar, unsigned target){
    unsigned spins = 0;
    while(ld_acquire_u32(bar) < target){
        spins++;
        if(spins > GRID_BARRIER_SPIN_LIMIT || ((spins & 63u) == 0u && ld_acquire_u32(bar + 2) != 0u)){ atomicExch(bar + 2, 1u); return false; }
    }
    return true;
}
// by one thread of every CTA, after its last barrier: the last of the `ctas` CTAs clears the slot for its next launch
__device__ __forceinline__ void grid_barrier_leave(unsigned* bar, unsigned ctas){
    const unsigned old = atomicAdd(bar + 1, 1u);
    if(old == ctas - 1){ bar[0] = 0u; bar[1] = 0u; __threadfence(); }
}

}  // namespace b200rl
