// Dynamic shared memory of a kernel launch
#pragma once
#include <cuda_runtime.h>

namespace lcg {

// Let kernel fn have `bytes` of dynamic shared memory; cudaErrorInvalidValue if no
// block can. The limit is one per process, kernel and device, shared by all threads:
// it is only ever raised, to the most a block can have, so that a call with short rows
// does not lower it between another thread's call and its launch. Up to 48 KB, less
// a kernel's static shared memory (below 1 KB here), need no limit of their own.
inline cudaError_t allow_smem(const void *fn, size_t bytes) {
    if (bytes <= 47 * 1024) return cudaSuccess;
    int dev = 0, optin = 0;
    cudaFuncAttributes a;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, fn);
    if (e != cudaSuccess) return e;
    const int most = optin - (int)a.sharedSizeBytes;
    if (bytes > (size_t)most) return cudaErrorInvalidValue;
    return a.maxDynamicSharedSizeBytes >= most
               ? cudaSuccess
               : cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
}

}  // namespace lcg
