// Facts about the current device that every launch asks for.
#pragma once
#include <cuda_runtime.h>

#include <atomic>

#include "gpu/cuda_driver.hpp"

namespace cclx {
namespace gpu {

// SMs of the current device, asked of the runtime once per device
inline int device_sms() {
    static std::atomic<int> known[64];
    int dev = 0;
    CUDA_CHECK(cudaGetDevice(&dev));
    int n = dev < 64 ? known[dev].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        CUDA_CHECK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
        if (dev < 64)
            known[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

} // namespace gpu
} // namespace cclx
