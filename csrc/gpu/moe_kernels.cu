// Expert-parallel helpers around the all-to-all: row gather in dispatch order
// and the combine step (un-permute + weighted sum of the top-k expert outputs).
//
// The reference offers alltoallv (src/coll/algorithms/alltoallv.cpp:112-751,
// alltoallv_kernel_* in src/kernels/kernels.cl:110-116) and leaves routing to the
// application; here the two memory-bound passes next to the exchange are
// kernels of the library so that the MoE layer is: route -> gather -> alltoallv
// -> expert FFN (tcgen05 GEMMs) -> alltoallv -> combine.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "capi/capi_common.hpp"
#include "core/log.hpp"
#include "gpu/cuda_driver.hpp"
#include "gpu/launch_util.cuh"

using namespace cclx;

namespace {

// out[i, :] = x[src_row[i], :]      (bf16 rows of `hidden` elements, hidden % 8 == 0)
__global__ void __launch_bounds__(256) gather_rows_kernel(const __nv_bfloat16* __restrict__ x,
                                                          const long long* __restrict__ src_row,
                                                          __nv_bfloat16* __restrict__ out, size_t n_rows,
                                                          int hidden) {
    const int packs = hidden / 8;
    for (size_t r = blockIdx.x; r < n_rows; r += gridDim.x) {
        const uint4* s = reinterpret_cast<const uint4*>(x + (size_t)src_row[r] * hidden);
        uint4* d = reinterpret_cast<uint4*>(out + r * hidden);
        for (int i = threadIdx.x; i < packs; i += blockDim.x)
            d[i] = s[i];
    }
}

// out[t, :] = sum_k w[t, k] * y[pos[t, k], :]   (fp32 accumulate, bf16 out)
__global__ void __launch_bounds__(256) combine_rows_kernel(const __nv_bfloat16* __restrict__ y,
                                                           const long long* __restrict__ pos,
                                                           const float* __restrict__ w,
                                                           __nv_bfloat16* __restrict__ out, size_t n_tokens, int topk,
                                                           int hidden) {
    const int packs = hidden / 8;
    for (size_t t = blockIdx.x; t < n_tokens; t += gridDim.x) {
        for (int i = threadIdx.x; i < packs; i += blockDim.x) {
            float acc[8] = { 0, 0, 0, 0, 0, 0, 0, 0 };
            for (int k = 0; k < topk; k++) {
                const float wk = w[t * topk + k];
                uint4 v = reinterpret_cast<const uint4*>(y + (size_t)pos[t * topk + k] * hidden)[i];
                const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&v);
#pragma unroll
                for (int e = 0; e < 8; e++)
                    acc[e] += wk * __bfloat162float(h[e]);
            }
            uint4 o;
            __nv_bfloat16* oh = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
            for (int e = 0; e < 8; e++)
                oh[e] = __float2bfloat16_rn(acc[e]);
            reinterpret_cast<uint4*>(out + t * hidden)[i] = o;
        }
    }
}

int blocks_for(size_t rows) {
    size_t cap = (size_t)gpu::device_sms() * 8;
    return (int)(rows < cap ? (rows ? rows : 1) : cap);
}

} // namespace

CCLX_API int cclx_moe_gather_rows(const void* x, const long long* src_row, void* out, size_t n_rows, int hidden,
                                  void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(hidden % 8 == 0, "hidden size must be a multiple of 8");
        if (n_rows == 0)
            return;
        gather_rows_kernel<<<blocks_for(n_rows), 256, 0, (cudaStream_t)stream>>>(
            (const __nv_bfloat16*)x, src_row, (__nv_bfloat16*)out, n_rows, hidden);
        CUDA_CHECK(cudaGetLastError());
    });
}

CCLX_API int cclx_moe_combine(const void* y, const long long* pos, const float* w, void* out, size_t n_tokens,
                              int topk, int hidden, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(hidden % 8 == 0, "hidden size must be a multiple of 8");
        if (n_tokens == 0)
            return;
        combine_rows_kernel<<<blocks_for(n_tokens), 256, 0, (cudaStream_t)stream>>>(
            (const __nv_bfloat16*)y, pos, w, (__nv_bfloat16*)out, n_tokens, topk, hidden);
        CUDA_CHECK(cudaGetLastError());
    });
}

// ---------------------------------------------------------------------------------------------
// Routing on the device: top-k experts per token with softmax weights over the chosen logits, the number of
// (token, slot) items per expert, and a permutation that groups the items by expert (with its inverse).  Two
// small kernels replace topk / softmax / bincount / argsort / scatter of an eager implementation (six launches
// and a sort).  Inside an expert's group the items stand in the order the atomics grant, which no consumer
// depends on: the combine step finds every item through `pos`, and an expert's rows are computed independently
// of their place.
// ---------------------------------------------------------------------------------------------
namespace {
constexpr int ROUTE_MAX_EXPERTS = 64;
constexpr int ROUTE_MAX_TOPK = 8;

// Top-k of one token's logits: ids, softmax weights over the chosen logits.  Ties go to the lower expert index (as
// torch.topk on a sorted scan would).  `pick(s, e)` is told every choice.  E: a bound of the number of experts for which
// the row is read once into registers, 0 for any number.
template <int E, class F>
__device__ __forceinline__ void route_token(const float* __restrict__ row, int n_experts, int topk, long long* __restrict__ idx,
                                            float* __restrict__ wts, F&& pick) {
    unsigned long long taken = 0; // a bit per expert
    int best[ROUTE_MAX_TOPK];
    float val[ROUTE_MAX_TOPK];
    __align__(16) float v[E > 0 ? E : 1];
    if constexpr (E > 0) {
        if (n_experts == E && (reinterpret_cast<uintptr_t>(row) & 15) == 0) {
#pragma unroll
            for (int e = 0; e < E; e += 4)
                *reinterpret_cast<float4*>(v + e) = *reinterpret_cast<const float4*>(row + e);
        }
        else {
#pragma unroll
            for (int e = 0; e < E; e++)
                if (e < n_experts)
                    v[e] = row[e];
        }
    }
#pragma unroll
    for (int s = 0; s < ROUTE_MAX_TOPK; s++) {
        if (s < topk) {
            int be = -1;
            float bv = 0.f;
            auto look = [&](int e, float x) {
                if (!(taken >> e & 1) && (be < 0 || x > bv)) {
                    be = e;
                    bv = x;
                }
            };
            if constexpr (E > 0) {
#pragma unroll
                for (int e = 0; e < E; e++)
                    if (e < n_experts)
                        look(e, v[e]);
            }
            else {
                for (int e = 0; e < n_experts; e++)
                    look(e, row[e]);
            }
            taken |= 1ull << be;
            best[s] = be;
            val[s] = bv;
        }
    }
    float sum = 0.f;
    const float vmax = val[0]; // the first pick is the maximum
#pragma unroll
    for (int s = 0; s < ROUTE_MAX_TOPK; s++)
        if (s < topk) {
            val[s] = __expf(val[s] - vmax);
            sum += val[s];
        }
#pragma unroll
    for (int s = 0; s < ROUTE_MAX_TOPK; s++)
        if (s < topk) {
            idx[s] = best[s];
            wts[s] = val[s] / sum;
            pick(s, best[s]);
        }
}

template <int E>
__global__ void __launch_bounds__(256)
    route_topk_kernel(const float* __restrict__ logits, int n_tokens, int n_experts, int topk, long long* __restrict__ idx,
                      float* __restrict__ wts, unsigned long long* __restrict__ counts) {
    __shared__ unsigned int hist[ROUTE_MAX_EXPERTS];
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x)
        hist[e] = 0;
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n_tokens)
        route_token<E>(logits + (size_t)t * n_experts, n_experts, topk, idx + (size_t)t * topk, wts + (size_t)t * topk,
                       [&](int, int e) { atomicAdd(&hist[e], 1u); });
    __syncthreads();
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x)
        if (hist[e])
            atomicAdd(&counts[e], (unsigned long long)hist[e]);
}

// The whole routing of a batch of up to ROUTE_ONE_BLOCK items in one block: selection, counts, offsets and placement with
// the counters in shared memory.  Latency is what it costs: 1024 tokens 4 us instead of two fills and two kernels (10 us).
constexpr int ROUTE_ONE_BLOCK = 8192;

template <int E>
__global__ void __launch_bounds__(1024)
    route_one_block_kernel(const float* __restrict__ logits, int n_tokens, int n_experts, int topk, long long* __restrict__ idx,
                           float* __restrict__ wts, unsigned long long* __restrict__ counts, long long* __restrict__ order,
                           long long* __restrict__ pos) {
    __shared__ unsigned int count[ROUTE_MAX_EXPERTS], offs[ROUTE_MAX_EXPERTS];
    __shared__ unsigned short ticket[ROUTE_ONE_BLOCK];
    __shared__ unsigned char expert[ROUTE_ONE_BLOCK];
    gpu::pdl_trigger();
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x)
        count[e] = 0;
    __syncthreads();
    gpu::pdl_wait(); // launched while the kernel in front still runs
    for (int t = threadIdx.x; t < n_tokens; t += blockDim.x)
        route_token<E>(logits + (size_t)t * n_experts, n_experts, topk, idx + (size_t)t * topk, wts + (size_t)t * topk,
                       [&](int s, int e) {
                           ticket[t * topk + s] = (unsigned short)atomicAdd(&count[e], 1u);
                           expert[t * topk + s] = (unsigned char)e;
                       });
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned acc = 0;
        for (int e = 0; e < n_experts; e++) {
            offs[e] = acc;
            acc += count[e];
        }
    }
    if (threadIdx.x < n_experts)
        counts[threadIdx.x] = count[threadIdx.x];
    __syncthreads();
    for (int i = threadIdx.x; i < n_tokens * topk; i += blockDim.x) {
        const unsigned p = offs[expert[i]] + ticket[i];
        order[p] = i;
        pos[i] = p;
    }
}

// cursor[e] starts at zero; item i = token * topk + slot lands at offset(expert) + ticket.  Tickets are drawn in
// shared memory first and every block asks the global counters once per expert (a million items on eight
// global counters would serialise on them).
__global__ void __launch_bounds__(256)
    route_place_kernel(const long long* __restrict__ idx, size_t n_items, int n_experts,
                       const unsigned long long* __restrict__ counts, unsigned int* __restrict__ cursor,
                       long long* __restrict__ order, long long* __restrict__ pos) {
    __shared__ unsigned long long offs[ROUTE_MAX_EXPERTS];
    __shared__ unsigned int local_n[ROUTE_MAX_EXPERTS], base[ROUTE_MAX_EXPERTS];
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x)
        local_n[e] = 0;
    if (threadIdx.x == 0) {
        unsigned long long acc = 0;
        for (int e = 0; e < n_experts; e++) {
            offs[e] = acc;
            acc += counts[e];
        }
    }
    __syncthreads();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    int e = -1;
    unsigned int ticket = 0;
    if (i < n_items) {
        e = (int)idx[i];
        ticket = atomicAdd(&local_n[e], 1u);
    }
    __syncthreads();
    for (int x = threadIdx.x; x < n_experts; x += blockDim.x)
        base[x] = local_n[x] ? atomicAdd(&cursor[x], local_n[x]) : 0u;
    __syncthreads();
    if (e >= 0) {
        const unsigned long long p = offs[e] + base[e] + ticket;
        order[p] = (long long)i;
        pos[i] = (long long)p;
    }
}
} // namespace

// items (token, slot) up to which one block does the whole routing
CCLX_API int cclx_moe_route_one_block() {
    return ROUTE_ONE_BLOCK;
}

// logits [n_tokens, n_experts] fp32 -> idx [n_tokens, topk] (int64), wts [n_tokens, topk] (fp32),
// counts [n_experts] (int64), order / pos [n_tokens * topk] (int64).  scratch: n_experts 32-bit words; right
// behind `counts` it is cleared together with them.
CCLX_API int cclx_moe_route(const float* logits, int n_tokens, int n_experts, int topk, long long* idx, float* wts,
                            long long* counts, long long* order, long long* pos, void* scratch, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(n_experts >= 1 && n_experts <= ROUTE_MAX_EXPERTS, "routing supports up to ", ROUTE_MAX_EXPERTS,
                         " experts");
        CCL_THROW_IF_NOT(topk >= 1 && topk <= ROUTE_MAX_TOPK && topk <= n_experts, "top-k must be between 1 and min(",
                         ROUTE_MAX_TOPK, ", experts)");
        cudaStream_t st = (cudaStream_t)stream;
        if (n_tokens > 0 && (size_t)n_tokens * topk <= ROUTE_ONE_BLOCK) {
            auto kernel = n_experts <= 8 ? route_one_block_kernel<8> : n_experts <= 16 ? route_one_block_kernel<16> : route_one_block_kernel<0>;
            const int threads = std::min(1024, (n_tokens + 31) / 32 * 32); // at least a warp; a thread per token
            gpu::launch_dependent(kernel, dim3(1), dim3(std::max(threads, 64)), 0, st, logits, n_tokens, n_experts, topk, idx, wts,
                                  (unsigned long long*)counts, order, pos);
            return;
        }
        if (scratch == (void*)(counts + n_experts))
            CUDA_CHECK(cudaMemsetAsync(counts, 0, (sizeof(long long) + sizeof(unsigned int)) * n_experts, st));
        else {
            CUDA_CHECK(cudaMemsetAsync(counts, 0, sizeof(long long) * n_experts, st));
            CUDA_CHECK(cudaMemsetAsync(scratch, 0, sizeof(unsigned int) * n_experts, st));
        }
        if (n_tokens == 0)
            return;
        auto topk_kernel = n_experts <= 8 ? route_topk_kernel<8> : n_experts <= 16 ? route_topk_kernel<16> : route_topk_kernel<0>;
        topk_kernel<<<(n_tokens + 255) / 256, 256, 0, st>>>(logits, n_tokens, n_experts, topk, idx, wts, (unsigned long long*)counts);
        CUDA_CHECK(cudaGetLastError());
        const size_t n_items = (size_t)n_tokens * topk;
        route_place_kernel<<<(unsigned)((n_items + 255) / 256), 256, 0, st>>>(
            idx, n_items, n_experts, (const unsigned long long*)counts, (unsigned int*)scratch, order, pos);
        CUDA_CHECK(cudaGetLastError());
    });
}

// ---------------------------------------------------------------------------------------------
// Fused dispatch and combine over peer memory: the all-to-all of an expert-parallel layer without
// staging buffers, send-side row gather or receive-side copies.
//
//   dispatch: every rank tells every peer how many rows it sends to each expert (a W x W table in
//             symmetric memory, written redundantly per block so that the per-block barrier is
//             enough), derives where its rows start inside each expert's receive buffer (ranks in
//             order), and stores row `order[i] / topk` of x straight into the owner's buffer.
//   combine : after the expert FFN wrote its output rows (same layout as the receive buffer) every
//             rank pulls the rows of its tokens from the owners with peer loads and forms the
//             weighted sum in fp32.
//
// The reference leaves both steps to alltoallv (src/coll/algorithms/alltoallv.cpp:112-751) around
// user kernels; on NVSwitch the rows can go directly where they are needed.
// ---------------------------------------------------------------------------------------------
#include "gpu/device/common.cuh"
#include "gpu/device_comm.hpp"

namespace {

using namespace cclx;
using namespace cclx::dev;

struct moe_rank_args {
    const __nv_bfloat16* x; // dispatch: [tokens, hidden] input rows | combine: unused
    const long long* order; // dispatch: (token, slot) pairs sorted by expert, as token * topk + slot
    const long long* send_counts; // dispatch: rows for every expert [world]
    const long long* expert; // combine: expert of every (token, slot) [tokens * topk]
    const long long* pos; // combine: place of (token, slot) in `order`
    const float* weight; // combine: routing weights [tokens * topk]
    __nv_bfloat16* out; // combine: [tokens, hidden]
    int* meta; // [0, W) first row of my block inside expert e's buffer, [W, 2W) prefix of send_counts,
               // [2W] rows this rank's expert received, [2W+1] 1 if some buffer overflowed
};

struct moe_args {
    moe_rank_args r0;
    const moe_rank_args* emu_tab;
    int emu;
    int topk;
    int hidden;
    size_t n_items; // tokens * topk
    size_t cap_rows; // rows of the receive / output buffers
    size_t buf_off; // heap offset of the receive buffer (dispatch) or of the expert output (combine)
    size_t cnt_off; // heap offset of the int32 table [blocks][W][W]
};

// The pieces of rows that a warp takes: warp, warp + nwarps, ... of row-major (row, piece) pairs, without a division per step.
struct piece_walk {
    size_t row;
    int piece, pieces;
    unsigned step_rows;
    int step_pieces;
    __device__ __forceinline__ piece_walk(unsigned warp, unsigned nwarps, int n) : pieces(n) {
        row = warp / n;
        piece = warp % n;
        step_rows = nwarps / n;
        step_pieces = nwarps % n;
    }
    __device__ __forceinline__ void next() {
        row += step_rows;
        piece += step_pieces;
        if (piece >= pieces) {
            piece -= pieces;
            row++;
        }
    }
};

__global__ void __launch_bounds__(512) moe_dispatch_kernel(const comm_dev* tab, moe_args a) {
    const int er = a.emu ? (int)blockIdx.y : 0;
    const comm_dev& c = tab[er];
    const moe_rank_args& ra = a.emu ? a.emu_tab[er] : a.r0;
    block_sync s;
    sync_begin(c, s);
    const int W = c.world;
    __shared__ int s_cnt[MAX_RANKS * MAX_RANKS], s_own[MAX_RANKS], s_dst[MAX_RANKS], s_pre[MAX_RANKS + 1], s_over;
    // my counts into every rank's table, slot of this block
    const size_t blk_words = (size_t)blockIdx.x * W * W;
    for (int i = threadIdx.x; i < W * W; i += blockDim.x) {
        const int p = i / W, e = i % W;
        const int v = (int)ra.send_counts[e];
        int* t = reinterpret_cast<int*>(c.heap[p] + a.cnt_off) + blk_words;
        t[c.rank * W + e] = v;
        if (p == 0)
            s_own[e] = v;
    }
    bool ok = peer_barrier(c, s);
    // The table is read by all threads at once and worked on in shared memory: one thread that walked it in global memory
    // waited W * W times for the L2, some 40 us for eight ranks, in every block.
    for (int i = threadIdx.x; i < W * W; i += blockDim.x)
        s_cnt[i] = __ldcv(reinterpret_cast<const int*>(c.heap[c.rank] + a.cnt_off) + blk_words + i);
    if (threadIdx.x == 0)
        s_over = 0;
    __syncthreads();
    if (threadIdx.x < W) {
        const int e = threadIdx.x;
        int off = 0, tot = 0, pre = 0;
        for (int q = 0; q < W; q++) {
            const int v = s_cnt[q * W + e];
            off += q < c.rank ? v : 0;
            tot += v;
            pre += q < e ? s_own[q] : 0;
        }
        s_dst[e] = off;
        s_pre[e] = pre;
        if (e == W - 1)
            s_pre[W] = pre + s_own[e];
        if (tot > (long long)a.cap_rows)
            s_over = 1;
        if (blockIdx.x == 0) {
            ra.meta[e] = off;
            ra.meta[W + e] = pre;
            if (e == c.rank)
                ra.meta[2 * W] = tot;
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0)
        ra.meta[2 * W + 1] = s_over;
    if (ok && !s_over) {
        // A warp moves up to 256 packs of a row at a time, eight per lane in flight, and fetches the index of its next row
        // meanwhile.  Pieces instead of rows: 2048 rows among 288 warps are 8 rounds for 7.1 rows each, their halves 15 for
        // 14.2 (the last barrier waited 8 us for the slowest of 50).
        const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
        const unsigned warp = blockIdx.x * wpb + (threadIdx.x >> 5), nwarps = gridDim.x * wpb;
        const int packs = a.hidden / 8;
        piece_walk w(warp, nwarps, (packs + 255) / 256);
        long long item = w.row < a.n_items ? ra.order[w.row] : 0;
        while (w.row < a.n_items) {
            const size_t i = w.row;
            const int first = w.piece * 256 + lane;
            const uint4* src = reinterpret_cast<const uint4*>(ra.x + (size_t)((unsigned)item / (unsigned)a.topk) * a.hidden);
            w.next();
            if (w.row < a.n_items)
                item = ra.order[w.row];
            int e = 0;
            while (e + 1 < W && (long long)i >= s_pre[e + 1])
                e++;
            const size_t row = (size_t)s_dst[e] + (i - (size_t)s_pre[e]);
            char* dst = c.heap[e] + a.buf_off + row * (size_t)a.hidden * 2;
            uint4 v[8];
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (first + k * 32 < packs)
                    v[k] = src[first + k * 32];
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (first + k * 32 < packs)
                    st16(dst + (size_t)(first + k * 32) * 16, v[k]);
        }
    }
    peer_barrier(c, s);
    sync_end(c, s, gridDim.x, 2, false);
}

__global__ void __launch_bounds__(512) moe_combine_kernel(const comm_dev* tab, moe_args a) {
    const int er = a.emu ? (int)blockIdx.y : 0;
    const comm_dev& c = tab[er];
    const moe_rank_args& ra = a.emu ? a.emu_tab[er] : a.r0;
    block_sync s;
    sync_begin(c, s);
    const int W = c.world;
    // every owner has finished its expert FFN (this launch is ordered after it on each rank's stream)
    bool ok = peer_barrier(c, s);
    if (ok) {
        const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
        const size_t warp = (size_t)blockIdx.x * wpb + (threadIdx.x >> 5), nwarps = (size_t)gridDim.x * wpb;
        const int packs = a.hidden / 8;
        const size_t tokens = a.n_items / a.topk;
        // Lane sl of a warp works out where the row of slot sl lies (expert, place, weight: three dependent loads) for the
        // warp's next token while the rows of this one are summed; four packs of two slots are in flight per lane.
        const int topk = a.topk;
        auto locate = [&](size_t t, int sl0, const char*& row, float& w) {
            row = nullptr;
            w = 0.f;
            if (t < tokens && sl0 + lane < topk) {
                const size_t f = t * topk + sl0 + lane;
                const int e = (int)ra.expert[f];
                const long long p = ra.pos[f];
                w = ra.weight[f];
                row = c.heap[e] + a.buf_off + (size_t)(ra.meta[e] + (p - ra.meta[W + e])) * (size_t)a.hidden * 2;
            }
        };
        const char* next_row;
        float next_w;
        locate(warp, 0, next_row, next_w);
        for (size_t t = warp; t < tokens; t += nwarps) {
            const char* my_row = next_row;
            float my_w = next_w;
            locate(t + nwarps, 0, next_row, next_w);
            for (int k0 = lane; k0 < (packs + 31) / 32 * 32; k0 += 128) {
                float acc[4][8] = {};
                for (int sl = 0; sl < topk; sl += 2) {
                    if (topk > 32 && sl % 32 == 0) // more slots than lanes
                        locate(t, sl, my_row, my_w);
                    uint4 v[2][4];
                    float w[2];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int from = min(sl + h, topk - 1) & 31;
                        const char* row = (const char*)__shfl_sync(0xffffffffu, (unsigned long long)my_row, from);
                        w[h] = __shfl_sync(0xffffffffu, my_w, from);
                        if (sl + h < topk)
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                if (k0 + k * 32 < packs)
                                    v[h][k] = ld_cv16(row + (size_t)(k0 + k * 32) * 16);
                    }
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        if (sl + h < topk)
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                if (k0 + k * 32 < packs) {
                                    const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&v[h][k]);
#pragma unroll
                                    for (int q = 0; q < 8; q++)
                                        acc[k][q] = fmaf(w[h], __bfloat162float(b[q]), acc[k][q]);
                                }
                }
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (k0 + k * 32 < packs) {
                        uint4 o;
                        __nv_bfloat16* oh = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
                        for (int q = 0; q < 8; q++)
                            oh[q] = __float2bfloat16_rn(acc[k][q]);
                        reinterpret_cast<uint4*>(ra.out + t * a.hidden)[k0 + k * 32] = o;
                    }
            }
        }
    }
    // nobody may overwrite its output rows (the next layer's FFN) before every reader is done
    peer_barrier(c, s);
    sync_end(c, s, gridDim.x, 2, false);
}

void launch_moe(gpu::device_comm& dc, bool dispatch, moe_args& a, const moe_rank_args* ra, int blocks,
                cudaStream_t st) {
    dc.check_status();
    blocks = blocks > 0 ? std::min(blocks, dc.max_blocks()) : std::min(dc.max_blocks(), 128);
    a.r0 = ra[0];
    if (dc.emulated()) {
        static_assert(sizeof(moe_rank_args) <= sizeof(dev::rank_args), "argument block too large");
        a.emu = 1;
        a.emu_tab = (const moe_rank_args*)dc.emu_table(dispatch ? gpu::device_comm::EMU_DISPATCH : gpu::device_comm::EMU_COMBINE, ra,
                                                       dc.world() * sizeof(moe_rank_args), st);
        const comm_dev* tab = dc.table();
        void* argv[] = { (void*)&tab, (void*)&a };
        dim3 grid(blocks, dc.world());
        CUDA_CHECK(cudaLaunchCooperativeKernel(dispatch ? (const void*)moe_dispatch_kernel : (const void*)moe_combine_kernel,
                                               grid, dim3(512), argv, 0, st));
    }
    else {
        a.emu = 0;
        a.emu_tab = nullptr;
        if (dispatch)
            moe_dispatch_kernel<<<blocks, 512, 0, st>>>(dc.table(), a);
        else
            moe_combine_kernel<<<blocks, 512, 0, st>>>(dc.table(), a);
        CUDA_CHECK(cudaGetLastError());
    }
}

} // namespace

// Arrays hold one pointer per entry: one entry in real mode, `world` entries in emulation mode.
// `recv_buf` / `cnt_table` are this rank's (entry 0's) symmetric allocations: [cap_rows, hidden] bf16 and
// at least 256 * world * world int32.  meta: 2 * world + 2 int32 per entry.
CCLX_API int cclx_moe_dispatch(void* h, const void* const* x, const long long* const* order,
                               const long long* const* send_counts, int* const* meta, size_t n_items, int topk,
                               int hidden, const void* recv_buf, size_t cap_rows, const void* cnt_table, int blocks,
                               void* stream) {
    return cclx::capi::guard([&] {
        gpu::device_comm* dc = (gpu::device_comm*)h;
        CCL_THROW_IF_NOT(hidden % 8 == 0 && topk >= 1, "hidden size must be a multiple of 8");
        const int entries = dc->emulated() ? dc->world() : 1;
        const int owner = dc->emulated() ? 0 : dc->rank();
        moe_args a{};
        a.topk = topk;
        a.hidden = hidden;
        a.n_items = n_items;
        a.cap_rows = cap_rows;
        a.buf_off = dc->symm_offset(recv_buf, owner);
        a.cnt_off = dc->symm_offset(cnt_table, owner);
        CCL_THROW_IF_NOT(a.buf_off != (size_t)-1 && a.cnt_off != (size_t)-1 && (a.buf_off & 15) == 0,
                         "the receive buffer and the count table must come from the symmetric heap");
        std::vector<moe_rank_args> ra(entries);
        for (int e = 0; e < entries; e++) {
            ra[e] = moe_rank_args{};
            ra[e].x = (const __nv_bfloat16*)x[e];
            ra[e].order = order[e];
            ra[e].send_counts = send_counts[e];
            ra[e].meta = meta[e];
        }
        launch_moe(*dc, true, a, ra.data(), blocks, (cudaStream_t)stream);
    });
}

CCLX_API int cclx_moe_combine_peer(void* h, const long long* const* expert, const long long* const* pos,
                                   const float* const* weight, void* const* out, int* const* meta, size_t n_items,
                                   int topk, int hidden, const void* expert_out, int blocks, void* stream) {
    return cclx::capi::guard([&] {
        gpu::device_comm* dc = (gpu::device_comm*)h;
        CCL_THROW_IF_NOT(hidden % 8 == 0 && topk >= 1, "hidden size must be a multiple of 8");
        const int entries = dc->emulated() ? dc->world() : 1;
        const int owner = dc->emulated() ? 0 : dc->rank();
        moe_args a{};
        a.topk = topk;
        a.hidden = hidden;
        a.n_items = n_items;
        a.buf_off = dc->symm_offset(expert_out, owner);
        CCL_THROW_IF_NOT(a.buf_off != (size_t)-1 && (a.buf_off & 15) == 0,
                         "the expert output must come from the symmetric heap");
        std::vector<moe_rank_args> ra(entries);
        for (int e = 0; e < entries; e++) {
            ra[e] = moe_rank_args{};
            ra[e].expert = expert[e];
            ra[e].pos = pos[e];
            ra[e].weight = weight[e];
            ra[e].out = (__nv_bfloat16*)out[e];
            ra[e].meta = meta[e];
        }
        launch_moe(*dc, false, a, ra.data(), blocks, (cudaStream_t)stream);
    });
}
