// Stores of bf16 rows from registers where every lane of a warp holds consecutive columns of a row of its own, as tcgen05.ld leaves
// them, in whole 32-byte sectors.  Optionally lanes trade sectors first, so that two or four neighbours write 64 or 128 contiguous
// bytes of one row: fewer lines per instruction, for 32 exchanges per 64 columns.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace cclx {
namespace gpu {

__device__ __forceinline__ void st_8(__nv_bfloat16* p, const uint32_t* w) { // 8 columns
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void st_16(__nv_bfloat16* p, const uint32_t* w) { // 16 columns, a whole sector
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

// N words of a lane in two halves: afterwards the lane whose bit `bit` is clear holds the first half of its own words and, behind it,
// the first of its partner's; the other lane the second halves, its partner's first.
template <int N>
__device__ __forceinline__ void trade(uint32_t* w, int lane, int bit) {
    const bool up = lane & bit;
#pragma unroll
    for (int k = 0; k < N / 2; k++) {
        const uint32_t lo = w[k], hi = w[N / 2 + k];
        const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? lo : hi, bit);
        w[k] = up ? got : lo;
        w[N / 2 + k] = up ? hi : got;
    }
}

// 32 or 64 columns per lane (16 or 32 words) of rows `row0` + lane from column `col` on into a matrix [M, N], N a multiple of 16 and
// its base 32-byte aligned.  Whole warps.
template <int W>
__device__ __forceinline__ void store_rows(__nv_bfloat16* m, int M, int N, int row0, int col, int lane, uint32_t (&w)[W]) {
    static_assert(W == 16 || W == 32, "two or four sectors per lane");
    if constexpr (W == 32) {
        trade<32>(w, lane, 2); // now halves of 32 columns: of row (lane & ~2), of row (lane | 2)
        trade<16>(w, lane, 1);
        trade<16>(w + 16, lane, 1);
        const int c = col + 16 * (lane & 3);
#pragma unroll
        for (int i = 0; i < 4; i++) { // rows 0, 1, 2, 3 of the four lanes
            const int r = row0 + (lane & ~3) + i;
            if (r < M && c < N)
                st_16(m + (size_t)r * N + c, w + 8 * i);
        }
    }
    else {
        trade<16>(w, lane, 1);
        const int c = col + 16 * (lane & 1);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int r = row0 + (lane & ~1) + i;
            if (r < M && c < N)
                st_16(m + (size_t)r * N + c, w + 8 * i);
        }
    }
}

} // namespace gpu
} // namespace cclx
