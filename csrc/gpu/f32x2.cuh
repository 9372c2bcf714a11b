// Pairs of fp32 values: one instruction adds or multiplies both (fma.rn.f32x2 and relatives), and the conversions
// between them and packs of eight bf16 values.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cclx {
namespace gpu {

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpair(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void unpack4x2(const uint4& u, f32x2 (&x)[4]) {
    const uint32_t w[4] = { u.x, u.y, u.z, u.w };
#pragma unroll
    for (int i = 0; i < 4; i++) // bf16 is the upper half of an fp32 word
        x[i] = pair(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}
__device__ __forceinline__ uint4 pack4x2(const f32x2 (&x)[4]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float lo, hi;
        unpair(x[i], lo, hi);
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

} // namespace gpu
} // namespace cclx
