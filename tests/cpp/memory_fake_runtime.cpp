// csrc/memory.cu over a fake of the CUDA runtime (no GPU): which calls the
// release of a handle's buffer makes when some of them are refused.
//   memory_fake_runtime <scenario>: prints the calls in order and "done".
#include <cstdio>
#include <cstring>
#include <string>

#include "memory.h"

namespace {
std::string scenario;
cudaStreamCaptureMode mode = cudaStreamCaptureModeGlobal;  // of the thread
cudaError_t last = cudaSuccess;
bool broken = false;  // the runtime is gone
bool armed = false;   // the scenario's failures begin

bool is(const char* s) { return armed && scenario == s; }
cudaError_t say(const char* call, cudaError_t e) {
    if (armed) std::printf("%s%s\n", call, e == cudaSuccess ? "" : " refused");
    if (e != cudaSuccess) last = e;
    return e;
}
// A capture in the global mode is open in another thread: calls that are unsafe
// beside it are refused unless this thread's mode is relaxed.
cudaError_t unsafe(const char* call) {
    const bool captured = is("capture") || scenario == "first";
    return say(call, captured && mode != cudaStreamCaptureModeRelaxed ? cudaErrorStreamCaptureUnsupported
                     : is("no_wait")                                  ? cudaErrorMemoryAllocation
                                                                      : cudaSuccess);
}
int block[4];
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return broken ? say("cudaGetDevice", cudaErrorCudartUnloading) : cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return broken ? say("cudaSetDevice", cudaErrorCudartUnloading) : cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t) {
    *p = block;
    return unsafe("cudaMalloc");
}
cudaError_t cudaFree(void*) { return unsafe("cudaFree"); }
cudaError_t cudaDeviceSynchronize() {  // refused beside any capture
    return say("cudaDeviceSynchronize",
               is("capture") || is("no_wait") ? cudaErrorStreamCaptureUnsupported : cudaSuccess);
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t, cudaStream_t) {
    *p = block + 1;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void*, cudaStream_t) {
    return broken ? say("cudaFreeAsync", cudaErrorCudartUnloading) : unsafe("cudaFreeAsync");
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
    *p = reinterpret_cast<cudaMemPool_t>(block + 2);
    return unsafe("cudaMemPoolCreate");
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(block + 3);
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
    std::swap(*m, mode);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
}

int main(int, char** argv) {
    scenario = argv[1];
    try {
        spc5cuda::Owned buf;
        buf.alloc(64);
        armed = true;
        broken = scenario == "unloading";
    } catch (const spc5cuda::Error& e) {
        std::printf("error: %s\n", e.what());
    }
    std::printf("mode %s\n", mode == cudaStreamCaptureModeGlobal ? "as before" : "changed");
    std::printf("last error %d\n", int(last));
    std::printf("done\n");
    return 0;
}
