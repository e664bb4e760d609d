// error.cuh -- CUDA runtime errors as exceptions that carry an MPS_ERR_* code.
#pragma once

#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "../../include/mps_b200.h"

namespace mps {

struct CudaError : std::runtime_error {
    int code;
    CudaError(const std::string &m, int c) : std::runtime_error(m), code(c) {}
};

// The error is thrown, so it does not stay behind for the next call's check.
#define MPS_CUDA(call)                                                                         \
    do {                                                                                       \
        cudaError_t e_ = (call);                                                               \
        if (e_ != cudaSuccess) {                                                               \
            (void)cudaGetLastError();                                                          \
            throw ::mps::CudaError(std::string(#call) + ": " + cudaGetErrorString(e_),         \
                                   e_ == cudaErrorMemoryAllocation ? MPS_ERR_OOM : MPS_ERR_CUDA); \
        }                                                                                      \
    } while (0)

}  // namespace mps
