// launch_limits.h — the dynamic shared memory that a kernel's launches may ask for.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace sky {

// Lets `kernel` be launched with `bytes` of dynamic shared memory.  The limit
// belongs to the kernel, not to the launch, and host threads with scenes of
// different sizes launch the same kernel: every one of them sets the device's
// maximum, so that none lowers the limit between another's setting and its
// launch (a launch above the maximum is refused by the launch itself).  The
// kernels have no static shared memory.
inline cudaError_t allow_shared_memory(const void* kernel, size_t bytes) {
    if (bytes <= 48u * 1024u) return cudaSuccess;
    int dev = 0, most = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    return e;
}

}  // namespace sky
