// smemlimit.cuh -- a kernel's limit of dynamic shared memory.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace dg {

// Dynamic shared memory a launch of `kernel` may ask for: `most`, the same on
// every call.  48 KB, less the kernel's static arrays (at most `held`), need no
// asking.  The limit belongs to the
// function, not to the launch, so a limit of this launch's own size would fail
// another thread's larger launch between its own call and its launch.
inline cudaError_t allow_smem(const void *kernel, size_t bytes, size_t most, size_t held)
{
    if (bytes + held <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes > most ? bytes : most));
}

}  // namespace dg
