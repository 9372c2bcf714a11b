// Token and position embedding of the decoder models: the sum of both rows in one pass, and the gradients added straight
// into the tables' gradient buffers in a fixed order, without sorting the tokens and without a dense gradient tensor of
// the table's size (the stock backward took a radix sort, a 103 MB fill and two 309 MB additions per step).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "capi/capi_common.hpp"
#include "core/log.hpp"
#include "gpu/cuda_driver.hpp"
#include "gpu/f32x2.cuh"
#include "gpu/launch_util.cuh"

using namespace cclx;
using namespace cclx::gpu;

namespace {

// out[i] = tokens[idx[i]] + positions[i % S]; one thread per 16-byte pack
__global__ void __launch_bounds__(128) embed_fwd_kernel(const long long* __restrict__ idx, const uint4* __restrict__ tokens,
                                                        const uint4* __restrict__ positions, uint4* __restrict__ out, size_t n,
                                                        int S, int table_rows, int packs) {
    const size_t i = (size_t)blockIdx.x * 128 + threadIdx.x;
    const size_t row = i / packs;
    if (row >= n)
        return;
    const int p = (int)(i - row * packs);
    f32x2 a[4], b[4];
    // an id outside the table reads nothing and makes its row NaN
    const bool ok = (unsigned long long)idx[row] < (unsigned long long)table_rows;
    unpack4x2(ok ? tokens[(size_t)idx[row] * packs + p] : make_uint4(~0u, ~0u, ~0u, ~0u), a);
    unpack4x2(positions[(row % S) * packs + p], b);
#pragma unroll
    for (int e = 0; e < 4; e++)
        a[e] = add2(a[e], b[e]);
    out[i] = pack4x2(a);
}

// Gradient of the token table.  A warp takes one position; if no earlier position has the same token it owns the token,
// lists all its positions in index order and adds the sum of their gradient rows (fp32) to the token's row, once.  The
// search runs over the ids in shared memory, 128 per step: n^2 / 128 steps, 5 us of the chip at 8192 positions, which is
// why longer batches take another way.  Rows are fetched eight at a time: a frequent token has hundreds.
constexpr int EMBED_MAX_IDS = 16384;
constexpr int EMBED_WARPS = 16;
constexpr int EMBED_LIST = 1024; // positions of one token summed between two updates of its row

__global__ void __launch_bounds__(EMBED_WARPS * 32)
    embed_bwd_kernel(const long long* __restrict__ idx, const uint4* __restrict__ dx, uint4* __restrict__ grad, int n, int table_rows,
                     int packs) {
    extern __shared__ int ids[]; // -1: no token of the table, or behind the end; then one list per warp
    const int padded = (n + 127) / 128 * 128;
    for (int i = threadIdx.x; i < padded; i += blockDim.x)
        ids[i] = i < n && (unsigned long long)idx[i] < (unsigned long long)table_rows ? (int)idx[i] : -1;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int4* ids4 = reinterpret_cast<const int4*>(ids);
    unsigned short* list = reinterpret_cast<unsigned short*>(ids + padded) + warp * EMBED_LIST;
    const int pos = blockIdx.x * EMBED_WARPS + warp;
    if (pos >= n || ids[pos] < 0)
        return;
    const int tok = ids[pos];
    for (int c = 0; c < pos; c += 128) {
        const int4 q = ids4[c / 4 + lane];
        const int j = c + lane * 4;
        if (__any_sync(0xffffffffu, (q.x == tok && j < pos) || (q.y == tok && j + 1 < pos) || (q.z == tok && j + 2 < pos) ||
                                        (q.w == tok && j + 3 < pos)))
            return; // an earlier position owns the token
    }
    uint4* out = grad + (size_t)tok * packs;
    int held = 0;
    auto add_listed = [&] {
        __syncwarp();
        for (int p = lane; p < packs; p += 32) {
            f32x2 acc[4];
            unpack4x2(out[p], acc);
            for (int k0 = 0; k0 < held; k0 += 8) {
                uint4 u[8];
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k0 + k < held)
                        u[k] = dx[(size_t)list[k0 + k] * packs + p];
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k0 + k < held) {
                        f32x2 a[4];
                        unpack4x2(u[k], a);
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            acc[e] = add2(acc[e], a[e]);
                    }
            }
            out[p] = pack4x2(acc);
        }
        held = 0;
        __syncwarp();
    };
    for (int c = pos / 128 * 128; c < padded; c += 128) {
        const int4 q = ids4[c / 4 + lane];
        const int j = c + lane * 4;
        const unsigned mine = (q.x == tok && j >= pos ? 1u : 0u) | (q.y == tok && j + 1 >= pos ? 2u : 0u) |
                              (q.z == tok && j + 2 >= pos ? 4u : 0u) | (q.w == tok && j + 3 >= pos ? 8u : 0u);
        unsigned lanes = __ballot_sync(0xffffffffu, mine != 0);
        if (!lanes)
            continue;
        if (held > EMBED_LIST - 128)
            add_listed();
        for (; lanes; lanes &= lanes - 1) { // in index order
            const int l = __ffs(lanes) - 1;
            const unsigned w = __shfl_sync(0xffffffffu, mine, l);
            for (int k = 0; k < 4; k++)
                if (w >> k & 1) {
                    if (lane == 0)
                        list[held] = (unsigned short)(c + l * 4 + k);
                    held++;
                }
        }
    }
    add_listed();
}

// gradient of the position table: row s (+)= the sum over the batch; rows behind S are cleared unless `add`
__global__ void __launch_bounds__(128) embed_pos_bwd_kernel(const uint4* __restrict__ dx, uint4* __restrict__ grad, int B, int S,
                                                            int table_rows, int packs, int add) {
    const size_t i = (size_t)blockIdx.x * 128 + threadIdx.x;
    const int s = (int)(i / packs);
    if (s >= (add ? S : table_rows))
        return;
    f32x2 acc[4] = { 0, 0, 0, 0 };
    if (s < S)
        for (int b0 = 0; b0 < B; b0 += 8) {
            uint4 u[8];
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (b0 + k < B)
                    u[k] = dx[(size_t)(b0 + k) * S * packs + i];
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (b0 + k < B) {
                    f32x2 a[4];
                    unpack4x2(u[k], a);
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        acc[e] = add2(acc[e], a[e]);
                }
        }
    if (add) {
        f32x2 a[4];
        unpack4x2(grad[i], a);
#pragma unroll
        for (int e = 0; e < 4; e++)
            acc[e] = add2(acc[e], a[e]);
    }
    grad[i] = pack4x2(acc);
}

} // namespace

// out[b, s, :] = tokens[idx[b, s], :] + positions[s, :]; bf16, D a multiple of 8
CCLX_API int cclx_embed_fwd(const long long* idx, const void* tokens, const void* positions, void* out, size_t n, int S,
                            int table_rows, int D, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(D % 8 == 0 && S > 0, "embedding rows must be whole 16-byte packs");
        const size_t total = n * (size_t)(D / 8);
        if (total == 0)
            return;
        embed_fwd_kernel<<<(unsigned)((total + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
            idx, (const uint4*)tokens, (const uint4*)positions, (uint4*)out, n, S, table_rows, D / 8);
        CUDA_CHECK(cudaGetLastError());
    });
}

// positions of a batch that cclx_embed_bwd takes
CCLX_API int cclx_embed_bwd_max_ids() {
    return EMBED_MAX_IDS;
}

// token_grad[idx[i], :] += dx[i, :] (ids outside the table are skipped), pos_grad[s, :] (+)= sum over the batch of dx[b, s, :]
CCLX_API int cclx_embed_bwd(const long long* idx, const void* dx, void* token_grad, void* pos_grad, int add_pos, int B, int S,
                            int token_rows, int pos_rows, int D, void* stream) {
    return cclx::capi::guard([&] {
        const int n = B * S, packs = D / 8;
        CCL_THROW_IF_NOT(D % 8 == 0 && n <= EMBED_MAX_IDS, "unsupported embedding gradient: ", n, " x ", D);
        cudaStream_t st = (cudaStream_t)stream;
        if (n > 0) {
            constexpr size_t lists = EMBED_WARPS * EMBED_LIST * sizeof(unsigned short);
            allow_smem<embed_bwd_kernel>(EMBED_MAX_IDS * 4 + lists);
            embed_bwd_kernel<<<(n + EMBED_WARPS - 1) / EMBED_WARPS, EMBED_WARPS * 32, (size_t)(n + 127) / 128 * 128 * 4 + lists,
                               st>>>(idx, (const uint4*)dx, (uint4*)token_grad, n, token_rows, packs);
            CUDA_CHECK(cudaGetLastError());
        }
        const size_t rows = add_pos ? S : pos_rows;
        if (rows > 0) {
            embed_pos_bwd_kernel<<<(unsigned)((rows * packs + 127) / 128), 128, 0, st>>>((const uint4*)dx, (uint4*)pos_grad, B, S,
                                                                                        pos_rows, packs, add_pos);
            CUDA_CHECK(cudaGetLastError());
        }
    });
}
