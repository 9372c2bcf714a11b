// 16-byte asynchronous copies from global to shared memory (cp.async).  A thread that reads back only what it copied
// itself needs no barrier: waiting for its own groups is enough, and no wait can last longer than the copies.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace cclx {
namespace gpu {

// `on` == false fills the 16 bytes with zeros and reads nothing
__device__ __forceinline__ void copy16_async(void* smem, const void* gmem, bool on) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(gmem), "r"(on ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copy_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

} // namespace gpu
} // namespace cclx
