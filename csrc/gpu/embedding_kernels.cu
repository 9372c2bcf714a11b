// Token and position embedding of the decoder models: the sum of both rows in one pass, and the gradients added straight
// into the tables' gradient buffers in a fixed order, without sorting the tokens and without a dense gradient tensor of
// the table's size (the stock backward took a radix sort, a 103 MB fill and two 309 MB additions per step).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "capi/capi_common.hpp"
#include "core/log.hpp"
#include "gpu/cuda_driver.hpp"
#include "gpu/f32x2.cuh"
#include "gpu/launch_util.cuh"

using namespace cclx;
using namespace cclx::gpu;

namespace {

// Word in mapped host memory that a kernel sets when it meets an id outside the table.  The host looks at it without waiting, so
// an error is reported by a later call.
int* bad_id_word() {
    static std::once_flag once;
    static int* word = nullptr;
    std::call_once(once, [] {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed; // an allocation is allowed beside this thread's capture
        CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode));
        const cudaError_t e = cudaHostAlloc((void**)&word, 64, cudaHostAllocMapped | cudaHostAllocPortable);
        CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode));
        CUDA_CHECK(e);
        *word = 0;
    });
    return word;
}

// out[i] = tokens[idx[i]] + positions[i % S]; one thread per 16-byte pack
__global__ void __launch_bounds__(128) embed_fwd_kernel(const long long* __restrict__ idx, const uint4* __restrict__ tokens,
                                                        const uint4* __restrict__ positions, uint4* __restrict__ out, size_t n,
                                                        int S, int table_rows, int packs, volatile int* bad_id) {
    const size_t i = (size_t)blockIdx.x * 128 + threadIdx.x;
    const size_t row = i / packs;
    if (row >= n)
        return;
    const int p = (int)(i - row * packs);
    f32x2 a[4], b[4];
    // an id outside the table reads nothing, makes its row NaN and is reported
    const bool ok = (unsigned long long)idx[row] < (unsigned long long)table_rows;
    if (!ok && p == 0)
        *bad_id = 1;
    unpack4x2(ok ? tokens[(size_t)idx[row] * packs + p] : make_uint4(~0u, ~0u, ~0u, ~0u), a);
    unpack4x2(positions[(row % S) * packs + p], b);
#pragma unroll
    for (int e = 0; e < 4; e++)
        a[e] = add2(a[e], b[e]);
    out[i] = pack4x2(a);
}

// Gradient of the token table.  A warp takes one position; if no earlier position has the same token it owns the token, lists all
// its positions in index order and adds the sum of their gradient rows (fp32) to the token's row, once.  Rows are fetched eight at
// a time.  The search runs over the ids in shared memory, 512 per step: n^2 / 512 steps, 5 us of the chip at 8192 positions, which
// is why longer batches take another way.  A token with more positions than the list holds is only flagged here and
// summed by embed_pos_bwd_kernel behind this one, 16 warps for every 256 columns: one warp needs 4.4 ms for a padded batch
// of 8192 positions of 1024 columns.
constexpr int EMBED_MAX_IDS = 16384;
constexpr int EMBED_STEP = 512; // ids per step of the search: four per lane and load, four loads in flight
constexpr int EMBED_WARPS = 16;
constexpr int EMBED_LIST = 64; // positions of a token that one warp sums

// acc += pack p of the rows list[from] ... list[to - 1], in that order
__device__ __forceinline__ void add_rows(const uint4* __restrict__ dx, int packs, int p, const unsigned short* list, int from, int to,
                                         f32x2 (&acc)[4]) {
    for (int k0 = from; k0 < to; k0 += 8) {
        uint4 u[8];
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k0 + k < to)
                u[k] = dx[(size_t)list[k0 + k] * packs + p];
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (k0 + k < to) {
                f32x2 a[4];
                unpack4x2(u[k], a);
#pragma unroll
                for (int e = 0; e < 4; e++)
                    acc[e] = add2(acc[e], a[e]);
            }
    }
}

__global__ void __launch_bounds__(EMBED_WARPS * 32)
    embed_bwd_kernel(const long long* __restrict__ idx, const uint4* __restrict__ dx, uint4* __restrict__ grad, int n, int table_rows,
                     int packs, unsigned char* __restrict__ frequent) {
    extern __shared__ int ids[]; // -1: no token of the table, or behind the end; then one list per warp
    const int padded = (n + EMBED_STEP - 1) / EMBED_STEP * EMBED_STEP;
    for (int i = threadIdx.x; i < padded; i += blockDim.x)
        ids[i] = i < n && (unsigned long long)idx[i] < (unsigned long long)table_rows ? (int)idx[i] : -1;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned short* list = reinterpret_cast<unsigned short*>(ids + padded) + warp * EMBED_LIST;
    const int pos = blockIdx.x * EMBED_WARPS + warp;
    if (pos >= n)
        return;
    if (lane == 0)
        frequent[pos] = 0;
    const int tok = ids[pos], own = pos / EMBED_STEP * EMBED_STEP; // the step that `pos` lies in
    if (tok < 0)
        return;
    // bit v * 4 + k of a lane: id c + v * 128 + lane * 4 + k is the token
    auto matches = [&](int c) {
        int4 q[4];
#pragma unroll
        for (int v = 0; v < 4; v++)
            q[v] = reinterpret_cast<const int4*>(ids + c)[v * 32 + lane];
        unsigned m = 0;
#pragma unroll
        for (int v = 0; v < 4; v++)
            m |= ((q[v].x == tok ? 1u : 0u) | (q[v].y == tok ? 2u : 0u) | (q[v].z == tok ? 4u : 0u) | (q[v].w == tok ? 8u : 0u)) << v * 4;
        return m;
    };
    unsigned earlier = 0; // bits of the ids of the own step in front of `pos`
#pragma unroll
    for (int v = 0; v < 4; v++)
        earlier |= ((1u << max(0, min(4, pos - own - v * 128 - lane * 4))) - 1) << v * 4;
    const unsigned here = matches(own);
    if (__any_sync(0xffffffffu, here & earlier))
        return; // an earlier position owns the token
    for (int c = 0; c < own; c += EMBED_STEP)
        if (__any_sync(0xffffffffu, matches(c)))
            return;
    int held = 0;
    for (int c = own; c < padded; c += EMBED_STEP) {
        const unsigned mine = c == own ? here & ~earlier : matches(c);
        const int found = __reduce_add_sync(0xffffffffu, __popc(mine));
        if (!found)
            continue;
        if (held + found > EMBED_LIST) {
            if (lane == 0)
                frequent[pos] = 1;
            return;
        }
#pragma unroll
        for (int v = 0; v < 4; v++)
            for (unsigned lanes = __ballot_sync(0xffffffffu, mine >> v * 4 & 15); lanes; lanes &= lanes - 1) { // in index order
                const int l = __ffs(lanes) - 1;
                const unsigned w = __shfl_sync(0xffffffffu, mine, l) >> v * 4;
                for (int k = 0; k < 4; k++)
                    if (w >> k & 1) {
                        if (lane == 0)
                            list[held] = (unsigned short)(c + v * 128 + l * 4 + k);
                        held++;
                    }
            }
    }
    __syncwarp();
    uint4* out = grad + (size_t)tok * packs;
    for (int p = lane; p < packs; p += 32) {
        f32x2 acc[4];
        unpack4x2(out[p], acc);
        add_rows(dx, packs, p, list, 0, held, acc);
        out[p] = pack4x2(acc);
    }
}

constexpr int EMBED_POS_THREADS = 512;

// exclusive prefix sum of `mine` over the block; `total`: of all threads.  Ends with a barrier in front of its next use.
__device__ __forceinline__ int block_prefix(int mine, int& total) {
    __shared__ int warps[EMBED_POS_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        incl += lane >= o ? v : 0;
    }
    if (lane == 31)
        warps[warp] = incl;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int i = 0; i < EMBED_POS_THREADS / 32; i++) {
        before += i < warp ? warps[i] : 0;
        total += warps[i];
    }
    __syncthreads();
    return before + incl - mine;
}

// The flagged tokens: block `b` of `blocks` takes every `blocks`-th of them, 32 packs of columns (`tile`).  The warps sum equal
// shares of the token's positions in order, shared memory joins them in order.
__device__ __forceinline__ void embed_frequent_tokens(const long long* __restrict__ idx, const unsigned char* __restrict__ frequent,
                                                      const uint4* __restrict__ dx, uint4* __restrict__ grad, int n, int packs, int b,
                                                      int blocks, int tile) {
    __shared__ __align__(16) unsigned char smem[EMBED_MAX_IDS * 2]; // the positions; afterwards the warps' sums
    __shared__ int first;
    unsigned short* list = reinterpret_cast<unsigned short*>(smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = EMBED_POS_THREADS / 32;
    const int share = (n + EMBED_POS_THREADS - 1) / EMBED_POS_THREADS, lo = threadIdx.x * share, hi = min(n, lo + share);
    int mine = 0, tokens, total;
    for (int i = lo; i < hi; i++)
        mine += frequent[i];
    const int at = block_prefix(mine, tokens);
    for (int f = b; f < tokens; f += blocks) {
        if (at <= f && f < at + mine)
            for (int i = lo, k = at; i < hi; i++)
                if (frequent[i] && k++ == f)
                    first = i;
        __syncthreads();
        const long long tok = idx[first];
        int have = 0;
        for (int i = lo; i < hi; i++)
            have += idx[i] == tok;
        int to = block_prefix(have, total);
        for (int i = lo; i < hi; i++)
            if (idx[i] == tok)
                list[to++] = (unsigned short)i;
        __syncthreads();
        const int p = tile * 32 + lane, per = (total + warps - 1) / warps;
        f32x2 acc[4] = { 0, 0, 0, 0 };
        if (p < packs)
            add_rows(dx, packs, p, list, min(total, warp * per), min(total, (warp + 1) * per), acc);
        __syncthreads();
        float2* sums = reinterpret_cast<float2*>(smem); // [warp][pack][4]
#pragma unroll
        for (int e = 0; e < 4; e++)
            unpair(acc[e], sums[(warp * 32 + lane) * 4 + e].x, sums[(warp * 32 + lane) * 4 + e].y);
        __syncthreads();
        if (threadIdx.x < 128 && tile * 32 + threadIdx.x / 4 < packs) { // two columns each
            __nv_bfloat162* out = reinterpret_cast<__nv_bfloat162*>(grad + (size_t)tok * packs + tile * 32) + threadIdx.x;
            float2 s = __bfloat1622float2(*out);
            for (int w = 0; w < warps; w++) {
                s.x += sums[w * 128 + threadIdx.x].x;
                s.y += sums[w * 128 + threadIdx.x].y;
            }
            *out = __floats2bfloat162_rn(s.x, s.y);
        }
        __syncthreads();
    }
}

// Gradient of the position table: row s (+)= the sum over the batch; rows behind S are cleared unless `add`.  The blocks from
// `pos_blocks` on sum the frequent tokens.
__global__ void __launch_bounds__(EMBED_POS_THREADS)
    embed_pos_bwd_kernel(const uint4* __restrict__ dx, uint4* __restrict__ grad, int B, int S, int table_rows, int packs, int add,
                         unsigned pos_blocks, const long long* __restrict__ idx, const unsigned char* __restrict__ frequent,
                         uint4* __restrict__ token_grad) {
    if (blockIdx.x >= pos_blocks) {
        const int tiles = (packs + 31) / 32, b = (int)(blockIdx.x - pos_blocks);
        embed_frequent_tokens(idx, frequent, dx, token_grad, B * S, packs, b / tiles, (int)(gridDim.x - pos_blocks) / tiles, b % tiles);
        return;
    }
    const size_t i = (size_t)blockIdx.x * EMBED_POS_THREADS + threadIdx.x;
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

// Whether a cclx_embed_fwd that has run met an id outside its table; clears the answer.
CCLX_API int cclx_embed_bad_id() {
    int bad = 0;
    const int rc = cclx::capi::guard([&] { bad = __atomic_exchange_n(bad_id_word(), 0, __ATOMIC_RELAXED); });
    return rc == 0 ? bad : 0;
}

// out[b, s, :] = tokens[idx[b, s], :] + positions[s, :]; bf16, D a multiple of 8
CCLX_API int cclx_embed_fwd(const long long* idx, const void* tokens, const void* positions, void* out, size_t n, int S,
                            int table_rows, int D, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(D % 8 == 0 && S > 0, "embedding rows must be whole 16-byte packs");
        const size_t total = n * (size_t)(D / 8);
        if (total == 0)
            return;
        embed_fwd_kernel<<<(unsigned)((total + 127) / 128), 128, 0, (cudaStream_t)stream>>>(
            idx, (const uint4*)tokens, (const uint4*)positions, (uint4*)out, n, S, table_rows, D / 8, bad_id_word());
        CUDA_CHECK(cudaGetLastError());
    });
}

// positions of a batch that cclx_embed_bwd takes
CCLX_API int cclx_embed_bwd_max_ids() {
    return EMBED_MAX_IDS;
}

// token_grad[idx[i], :] += dx[i, :] (ids outside the table are skipped), pos_grad[s, :] (+)= sum over the batch of dx[b, s, :].
// workspace: B * S bytes
CCLX_API int cclx_embed_bwd(const long long* idx, const void* dx, void* token_grad, void* pos_grad, int add_pos, int B, int S,
                            int token_rows, int pos_rows, int D, void* workspace, void* stream) {
    return cclx::capi::guard([&] {
        const int n = B * S, packs = D / 8;
        CCL_THROW_IF_NOT(D % 8 == 0 && n <= EMBED_MAX_IDS, "unsupported embedding gradient: ", n, " x ", D);
        cudaStream_t st = (cudaStream_t)stream;
        unsigned char* frequent = (unsigned char*)workspace;
        if (n > 0) {
            constexpr size_t lists = EMBED_WARPS * EMBED_LIST * sizeof(unsigned short);
            allow_smem<embed_bwd_kernel>(EMBED_MAX_IDS * 4 + lists);
            embed_bwd_kernel<<<(n + EMBED_WARPS - 1) / EMBED_WARPS, EMBED_WARPS * 32,
                               (size_t)(n + EMBED_STEP - 1) / EMBED_STEP * EMBED_STEP * 4 + lists, st>>>(
                idx, (const uint4*)dx, (uint4*)token_grad, n, token_rows, packs, frequent);
            CUDA_CHECK(cudaGetLastError());
        }
        const size_t rows = add_pos ? S : pos_rows;
        const unsigned pos_blocks = (unsigned)((rows * packs + EMBED_POS_THREADS - 1) / EMBED_POS_THREADS);
        // as many at once as there can be frequent tokens, up to 32
        const unsigned more = (unsigned)(std::min(n / (EMBED_LIST + 1), 32) * ((packs + 31) / 32));
        if (pos_blocks + more > 0) {
            embed_pos_bwd_kernel<<<pos_blocks + more, EMBED_POS_THREADS, 0, st>>>(
                (const uint4*)dx, (uint4*)pos_grad, B, S, pos_rows, packs, add_pos, pos_blocks, idx, frequent, (uint4*)token_grad);
            CUDA_CHECK(cudaGetLastError());
        }
    });
}
