// The grid-wide barrier of the cooperative kernels on its own: a launch some of whose CTAs never arrive, on a barrier that the library hands out.
#include "../../rl-tools_b200/csrc/grid_barrier.cuh"
using namespace b200rl;

__global__ void barrier_case_kernel(GridBarrier bar, int absent, int* passed){
    if((int)blockIdx.x >= absent){
        grid_barrier_arrive(bar);
        passed[blockIdx.x] = grid_barrier_wait(bar, gridDim.x) ? 1 : 0;
    }
    grid_barrier_leave(bar, gridDim.x);
}

extern "C" int barrier_case_take(GridBarrier* bar, void* stream){ return grid_barriers(1, (cudaStream_t)stream, bar); }
extern "C" int barrier_case_run(const GridBarrier* bar, int ctas, int absent, int* passed, void* stream){
    GridBarrier b = *bar;
    void* params[] = { &b, &absent, &passed };
    return (int)cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(barrier_case_kernel), dim3(ctas), dim3(1), params, 0, (cudaStream_t)stream);
}
extern "C" int barrier_case_words(const GridBarrier* bar, unsigned* words_host){ return (int)cudaMemcpy(words_host, bar->words, 4 * sizeof(unsigned), cudaMemcpyDeviceToHost); }
