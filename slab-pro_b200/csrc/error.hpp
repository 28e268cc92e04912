// The exception that the C entry points turn into a slab_status, and the check
// of a CUDA runtime call that throws it.
#pragma once

#include <cuda_runtime.h>

#include <string>

#include "slab_gpu.h"

namespace slab {

struct Error {
    slab_status code;
    std::string msg;
};

#define SLAB_CUDA(call)                                                                                         \
    do {                                                                                                        \
        cudaError_t e_ = (call);                                                                                \
        if (e_ != cudaSuccess)                                                                                  \
            throw ::slab::Error{e_ == cudaErrorMemoryAllocation ? SLAB_E_OOM : SLAB_E_CUDA,                     \
                                std::string(#call) + ": " + cudaGetErrorString(e_)};                            \
    } while (0)

}  // namespace slab
