// smemlimit.cuh -- a kernel's limit of dynamic shared memory.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace dg {

// Dynamic shared memory a launch of `kernel` may ask for: `most`, the same on
// every call.  48 KB, less the kernel's static arrays (at most `held`), need no
// asking.  The limit belongs to the
// function, not to the launch, so a limit of this launch's own size would fail
// another thread's larger launch between its own call and its launch.  The driver
// splits L1 and shared memory by that limit, so a limit above the launch's size
// asks for the largest shared part itself (one solve of N = 16384, leaf 128, rank
// 16: 81.2 us with a limit of the launch's size, 81.7 with the fixed limit alone or
// with the split asked for before it, 81.2 with the split asked for after it).
inline cudaError_t allow_smem(const void *kernel, size_t bytes, size_t most, size_t held)
{
    if (bytes + held <= 48 * 1024) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)(bytes > most ? bytes : most));
    return e != cudaSuccess ? e : cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                                       cudaSharedmemCarveoutMaxShared);
}

}  // namespace dg
