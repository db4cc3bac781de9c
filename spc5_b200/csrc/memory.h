// memory.h -- device memory of the library: per-call scratch and the handles'
// buffers (no device code).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "errors.h"

namespace spc5cuda {

// The library's memory pool on the current device (memory.cu): per-call scratch
// and the handles' buffers come from it.  It keeps up to 4 GiB of freed memory
// for the next allocation (mapping memory afresh for every buffer took most of
// a conversion's time) and gives the rest back.
cudaMemPool_t scratch_pool();
// A stream of the current device that only orders the pool's persistent
// buffers.
cudaStream_t alloc_stream();

// Gives a persistent buffer of device dev, whose allocation stream is s, back to
// the pool after all work of the device; keeps it out of the pool when it could
// not wait.
void give_back(void* p, int dev, cudaStream_t s) noexcept;

// Stream-ordered scratch.
struct PoolBuf {
    void* p = nullptr;
    size_t bytes = 0;
    cudaStream_t s;
    PoolBuf(size_t n, cudaStream_t st) : bytes(n), s(st) {
        SPC5_CUDA(cudaMallocFromPoolAsync(&p, n < 16 ? size_t(16) : n, scratch_pool(), st));
    }
    ~PoolBuf() {
        if (p) cudaFreeAsync(p, s);
    }
    PoolBuf(const PoolBuf&) = delete;
    PoolBuf& operator=(const PoolBuf&) = delete;
    template <class U>
    U* as() const { return static_cast<U*>(p); }
};
using DevBuf = PoolBuf;

// Persistent device buffer owned by a matrix handle.  alloc() returns memory
// that every stream may use; release() waits for the device first, as kernels
// on any stream may still use the buffer.
struct Owned {
    void* p = nullptr;
    size_t bytes = 0;
    int dev = 0;
    cudaStream_t s = nullptr;  // the device's allocation stream
    void alloc(size_t n) {
        release();
        if (n) {
            SPC5_CUDA(cudaGetDevice(&dev));
            s = alloc_stream();
            SPC5_CUDA(cudaMallocFromPoolAsync(&p, n, scratch_pool(), s));
            SPC5_CUDA(cudaStreamSynchronize(s));
        }
        bytes = n;
    }
    void release() noexcept {
        if (p) give_back(p, dev, s);
        p = nullptr;
        bytes = 0;
    }
    Owned() = default;
    Owned(const Owned&) = delete;
    Owned& operator=(const Owned&) = delete;
    Owned(Owned&& o) noexcept : p(o.p), bytes(o.bytes), dev(o.dev), s(o.s) {
        o.p = nullptr;
        o.bytes = 0;
    }
    Owned& operator=(Owned&& o) noexcept {
        if (this != &o) {
            release();
            p = o.p;
            bytes = o.bytes;
            dev = o.dev;
            s = o.s;
            o.p = nullptr;
            o.bytes = 0;
        }
        return *this;
    }
    ~Owned() { release(); }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

}  // namespace spc5cuda
