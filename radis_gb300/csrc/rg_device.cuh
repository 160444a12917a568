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

// The kernels of a spectrum are launched chained (programmatic dependent
// launch): the next one's launch is prepared while its predecessor runs, its
// CTAs start as soon as the predecessor's last ones have exited, and each waits
// in chain_begin until the predecessor's writes are visible.  All threads call
// it before they touch global memory that other kernels write (read by plain
// loads: the read-only path may be moved up across the wait).  A kernel
// exits only after its own wait, so what came before it is finished too.  Behind
// anything but a kernel (copies, memsets, events) it starts as usual.
// Against plain launches, spectra back to back: 10k lines 48.3 -> 41.6 us, 5M
// 125 -> 115, a dense band 207 -> 197.  Letting the next kernel in earlier
// (launch_dependents) only parks its CTAs on the SMs: right after the wait 44.9,
// 122.5 and 201 us, before the last part of the scatter and of the row kernel
// 44.4, 119.7 and 199.7.
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
static int launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
    return check_launch();
}

}  // namespace rg
