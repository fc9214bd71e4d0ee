// Errors of the CUDA runtime as the library's status codes.
#pragma once

#include <cuda_runtime.h>

#include "../../../include/mypbr_gpu.h"

namespace mypbr_dev {

// The status of a failed call; the message is kept for mypbr_last_error.
int cuda_fail(cudaError_t e, const char* what);

}  // namespace mypbr_dev

#define MYPBR_CUDA(call)                                       \
    do {                                                       \
        cudaError_t e_ = (call);                               \
        if (e_ != cudaSuccess)                                 \
            return ::mypbr_dev::cuda_fail(e_, #call);          \
    } while (0)
