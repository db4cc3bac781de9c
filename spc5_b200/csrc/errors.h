// errors.h -- the host layer's errors (no device code).
#pragma once

#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "spc5cuda.h"

namespace spc5cuda {

// Thrown inside the host layer, turned into a status code at the C ABI.
struct Error : std::runtime_error {
    spc5cuda_status status;
    Error(spc5cuda_status s, const std::string& what) : std::runtime_error(what), status(s) {}
};

inline void check_cuda(cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        throw Error(e == cudaErrorMemoryAllocation ? SPC5CUDA_ERR_NOMEM : SPC5CUDA_ERR_CUDA,
                    std::string(what) + ": " + cudaGetErrorString(e));
    }
}

#define SPC5_CUDA(call) ::spc5cuda::check_cuda((call), #call)

}  // namespace spc5cuda
