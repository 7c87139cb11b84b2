// Where the barriers of cooperative launches lie (grid_barrier.cuh), and the status of those whose wait ran into its limit.
#include "grid_barrier.cuh"
#include <mutex>

namespace b200rl {

// Two launches may use one barrier as long as they never run at the same time. Launches outside a capture take theirs round-robin: for two of them to meet, one
// would have to wait on its stream while BARRIER_RING others are issued and the last of them runs. A captured launch keeps its barrier for every replay, beside
// whatever runs then, so it gets one that nobody else is given; when those are used up, the caller takes the kernels that need none.
constexpr unsigned BARRIER_RING = 16384, BARRIER_CAPTURED = 16384;
static __device__ unsigned g_barriers[(BARRIER_RING + BARRIER_CAPTURED) * 4];

namespace {
struct DeviceBarriers { unsigned* words; unsigned* status_host; unsigned* status; unsigned next, next_captured; };
DeviceBarriers g_device[MAX_DEVICES] = {};
std::mutex g_mutex;
}

int grid_barriers(int count, cudaStream_t stream, GridBarrier* out){
    int dev = 0;
    int rc = current_device(&dev);
    if(rc) return rc;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    B200RL_CUDA_TRY(cudaStreamIsCapturing(stream, &capture));
    std::lock_guard<std::mutex> lock(g_mutex);
    DeviceBarriers& d = g_device[dev];
    if(d.words == nullptr){
        void* words = nullptr; void* host = nullptr; void* status = nullptr;
        B200RL_CUDA_TRY(cudaGetSymbolAddress(&words, g_barriers));
        // the first call may be a captured one: allocating host memory is no work of the stream's
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        B200RL_CUDA_TRY(cudaThreadExchangeStreamCaptureMode(&mode));
        cudaError_t e = cudaHostAlloc(&host, sizeof(unsigned), cudaHostAllocMapped | cudaHostAllocPortable);
        if(e == cudaSuccess) e = cudaHostGetDevicePointer(&status, host, 0);
        cudaThreadExchangeStreamCaptureMode(&mode);
        B200RL_CUDA_TRY(e);
        *static_cast<volatile unsigned*>(host) = 0u;
        d.status_host = static_cast<unsigned*>(host); d.status = static_cast<unsigned*>(status);
        d.words = static_cast<unsigned*>(words);
    }
    if(*static_cast<volatile unsigned*>(d.status_host) != 0u) return B200RL_ERR_DEVICE_FLAG;
    unsigned first = 0;
    if(capture == cudaStreamCaptureStatusNone){
        if(d.next + (unsigned)count > BARRIER_RING) d.next = 0;
        first = d.next;
        d.next += (unsigned)count;
    }
    else{
        if(d.next_captured + (unsigned)count > BARRIER_CAPTURED) return B200RL_ERR_UNSUPPORTED;
        first = BARRIER_RING + d.next_captured;
        d.next_captured += (unsigned)count;
    }
    for(int i = 0; i < count; i++) out[i] = GridBarrier{d.words + 4 * (first + i), d.status};
    return B200RL_OK;
}

int grid_barrier_status(unsigned* status){
    int dev = 0;
    const int rc = current_device(&dev);
    if(rc) return rc;
    std::lock_guard<std::mutex> lock(g_mutex);
    *status = g_device[dev].status_host ? *static_cast<volatile unsigned*>(g_device[dev].status_host) : 0u;
    return B200RL_OK;
}
int grid_barrier_clear(){
    int dev = 0;
    const int rc = current_device(&dev);
    if(rc) return rc;
    std::lock_guard<std::mutex> lock(g_mutex);
    if(g_device[dev].status_host) *static_cast<volatile unsigned*>(g_device[dev].status_host) = 0u;
    return B200RL_OK;
}

}  // namespace b200rl

// 0: no barrier of a cooperative launch on the current device ran into its limit since the last b200rl_device_error_clear
extern "C" int b200rl_cooperative_pass_status(int* status){
    using namespace b200rl;
    if(!status) return B200RL_ERR_INVALID_ARGUMENT;
    B200RL_CUDA_TRY(cudaDeviceSynchronize());
    unsigned word = 0;
    const int rc = grid_barrier_status(&word);
    *status = (int)word;
    return rc;
}
