// Launch helpers.
//
// Programmatic dependent launch: a kernel that is launched with launch_dependent() may start while the kernel in
// front of it on the stream still runs; it calls pdl_wait() before it touches anything that kernel wrote.  The
// earlier kernel calls pdl_trigger() once its blocks need not keep the later one from being scheduled.  What this
// hides is the launch latency and the prologue of short kernels (2 to 3 us of a 3 us kernel).
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <utility>

#include "gpu/cuda_driver.hpp"
#include "gpu/device_info.hpp"

namespace cclx {
namespace gpu {

__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void pdl_trigger() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
void launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...));
}

// dynamic shared memory above the default 48 KB, granted to the kernel once per device
template <auto KERNEL>
void allow_smem(size_t bytes) {
    static std::atomic<bool> done[64];
    int dev = 0;
    CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 64 && done[dev].load(std::memory_order_acquire))
        return;
    CUDA_CHECK(cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    if (dev < 64)
        done[dev].store(true, std::memory_order_release);
}

} // namespace gpu
} // namespace cclx
