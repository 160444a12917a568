// Helpers shared by the device translation units (rg_kernels.cu, rg_fft.cu).
#pragma once

#include <cuda_runtime.h>

#include <atomic>

#include "rg_internal.h"

namespace rg {

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// status of the launch just made (the CUDA error text is kept per thread)
int check_launch();

// Opt the kernel in to the largest dynamic shared memory the device allows
// next to the kernel's own static shared memory; checks that `need` fits.
// (first call per kernel: queries the attributes and sets the limit; later
// calls only compare `need` with the cached limit)
template <typename K>
static int allow_smem(K kernel, std::atomic<size_t>& avail_cache, size_t need) {
    size_t avail = avail_cache.load();
    if (!avail) {
        int dev = 0, optin = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return RG_ERR_CUDA;
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
            return RG_ERR_CUDA;
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return RG_ERR_CUDA;
        avail = (size_t)optin - fa.sharedSizeBytes;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)avail) != cudaSuccess)
            return RG_ERR_CUDA;
        avail_cache.store(avail);
    }
    return need > avail ? RG_ERR_RANGE : RG_OK;
}

#define ALLOW_SMEM(kernel, need)                          \
    do {                                                   \
        static std::atomic<size_t> avail_{0};              \
        int r_ = allow_smem(kernel, avail_, (need));       \
        if (r_ != RG_OK) return r_;                        \
    } while (0)

}  // namespace rg
