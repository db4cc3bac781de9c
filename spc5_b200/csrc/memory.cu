// memory.cu -- the library's memory pool per device, and the order in which the
// handles' buffers go back to it (memory.h).
#include "memory.h"

#include <stdint.h>

#include <cstring>
#include <mutex>

namespace spc5cuda {

namespace {

// The calling thread's captures, and those of other threads in the global mode,
// refuse calls that are unsafe beside them (cudaMalloc, cudaFree, cudaFreeAsync)
// and are spoilt by them; in this scope the calls are allowed, for memory that no
// capture uses.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Waits for all work on the current device, as freeing memory does: unlike
// cudaDeviceSynchronize(), that leaves a capture that is open on another stream
// alone.  False when the wait was refused.
bool wait_device() {
    void* p = nullptr;
    if (cudaMalloc(&p, 16) == cudaSuccess && cudaFree(p) == cudaSuccess) return true;
    cudaGetLastError();
    return cudaDeviceSynchronize() == cudaSuccess;
}

// One pool and one allocation stream per device for the process lifetime.
struct DeviceMemory {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    void* anchor = nullptr;  // keeps the memory mapped that wait_device() takes and frees
};

const DeviceMemory& device_memory() {
    static std::mutex mu;
    static DeviceMemory mem[64];
    constexpr uint64_t keep = uint64_t(4) << 30;
    int dev = 0;
    SPC5_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) throw Error(SPC5CUDA_ERR_UNSUPPORTED, "device index");
    std::lock_guard<std::mutex> lk(mu);
    DeviceMemory& m = mem[dev];
    if (!m.stream) {
        if (!m.pool) {
            cudaMemPoolProps props;
            std::memset(&props, 0, sizeof(props));
            props.allocType = cudaMemAllocationTypePinned;
            props.location.type = cudaMemLocationTypeDevice;
            props.location.id = dev;
            SPC5_CUDA(cudaMemPoolCreate(&m.pool, &props));
            uint64_t bytes = keep;
            SPC5_CUDA(cudaMemPoolSetAttribute(m.pool, cudaMemPoolAttrReleaseThreshold, &bytes));
        }
        if (!m.anchor) SPC5_CUDA(cudaMalloc(&m.anchor, 16));
        SPC5_CUDA(cudaStreamCreateWithFlags(&m.stream, cudaStreamNonBlocking));
    }
    return m;
}

}  // namespace

cudaMemPool_t scratch_pool() { return device_memory().pool; }
cudaStream_t alloc_stream() { return device_memory().stream; }

void give_back(void* p, int dev, cudaStream_t s) noexcept {
    int now = 0;
    if (cudaGetDevice(&now) != cudaSuccess) {  // the runtime unloads
        cudaGetLastError();
        return;
    }
    const RelaxedCapture relaxed;
    bool ok = now == dev || cudaSetDevice(dev) == cudaSuccess;
    ok = ok && wait_device() && cudaFreeAsync(p, s) == cudaSuccess;
    if (now != dev) cudaSetDevice(now);
    if (!ok) cudaGetLastError();  // not left for the next call's check to report
}

}  // namespace spc5cuda
