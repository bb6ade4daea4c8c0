// Copies and clears from the host that are complete when they return.
//
// cudaMemset is asynchronous to the host, and cudaMemcpy from pageable memory may
// return once its source has been staged.  Both run on the legacy stream, which
// orders them against default-stream work but not against kernels on a
// non-blocking stream: those are launched only after the wait here.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace glisser {

inline cudaError_t copy_to_device(void* dst, const void* src, size_t bytes)
{
    const cudaError_t e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
    return e == cudaSuccess ? cudaStreamSynchronize(nullptr) : e;
}

inline cudaError_t clear_on_device(void* dst, size_t bytes)
{
    const cudaError_t e = cudaMemset(dst, 0, bytes);
    return e == cudaSuccess ? cudaStreamSynchronize(nullptr) : e;
}

}  // namespace glisser
