// shared_limit.h -- how much dynamic shared memory a kernel may be launched with.
#pragma once
#include <cuda_runtime.h>

namespace ether {

// Lets `kernel` be launched with all the dynamic shared memory that a block can have beside the
// kernel's static arrays.  The limit belongs to the process, not to a context: where each context
// set its own need, two host threads could leave the smaller one's, and the other's launches were
// then refused (also where both read the limit first and only raise it).  One value from
// everybody leaves nothing to order.
inline cudaError_t allow_shared(const void *kernel) {
    int dev = 0, most = 0;
    cudaFuncAttributes fa;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, kernel);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes);
}

}  // namespace ether
