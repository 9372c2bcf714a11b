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
#include <type_traits>
#include <vector>

#include "capi/capi_common.hpp"
#include "core/log.hpp"
#include "gpu/cuda_driver.hpp"
#include "gpu/device/sm100_ptx.cuh"
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
namespace sm100 = cclx::sm100;
constexpr int ROUTE_MAX_EXPERTS = 64;
constexpr int ROUTE_MAX_TOPK = 8;

// Top-k of one token's logits: ids, softmax weights over the chosen logits.  Ties go to the lower expert index (as
// torch.topk on a sorted scan would).  `pick(s, e)` is told every choice.  E: a bound of the number of experts for which
// the row is read once into registers, 0 for any number.
template <int E, class F>
__device__ __forceinline__ void route_token(const float* row, int n_experts, int topk, long long* __restrict__ idx,
                                            float* __restrict__ wts, F&& pick) {
    std::conditional_t<(E > 0 && E <= 32), unsigned, unsigned long long> taken = 0; // a bit per expert
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
            taken |= (decltype(taken))1 << be;
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

// The whole routing of a batch of up to ROUTE_ONE_LAUNCH items in one launch: selection, counts, offsets and placement with the
// counters in shared memory, in one block or in a cluster of C that exchange their counts.  Latency is what it costs; the selection
// takes some 300 instructions per token, 2.5 us for 1024 tokens on one SM.  From 512 tokens on a cluster is
// faster: 1024 tokens among 8 experts, top-2, 2.5 us instead of 4.0 in a chain of such calls, 4096 tokens 3.4 instead of 12.0; 256
// tokens take 2.2 in one block.
constexpr int ROUTE_ONE_LAUNCH = 8192;
constexpr int ROUTE_CLUSTER = 8;
constexpr int ROUTE_CLUSTER_TOKENS = 512; // from so many tokens on

template <int E, int C>
__global__ void __launch_bounds__(1024)
    route_one_launch_kernel(const float* logits, int n_tokens, int n_experts, int topk, long long* __restrict__ idx,
                           float* __restrict__ wts, unsigned long long* __restrict__ counts, long long* __restrict__ order,
                           long long* __restrict__ pos) {
    constexpr int ITEMS = C > 1 ? ROUTE_ONE_LAUNCH / C + ROUTE_MAX_TOPK : ROUTE_CLUSTER_TOKENS * ROUTE_MAX_TOPK;
    __shared__ unsigned int count[ROUTE_MAX_EXPERTS], offs[ROUTE_MAX_EXPERTS], all[C][ROUTE_MAX_EXPERTS];
    __shared__ unsigned short ticket[ITEMS];
    __shared__ unsigned char expert[ITEMS];
    gpu::pdl_trigger();
    if constexpr (C > 1)
        sm100::cluster_arrive_relaxed(); // this block runs: the others may write its shared memory
    const int lane = threadIdx.x & 31, me = C > 1 ? (int)blockIdx.x : 0;
    const int per = (n_tokens + C - 1) / C, t0 = me * per, n = max(0, min(per, n_tokens - t0)); // tokens of this block
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x)
        count[e] = 0;
    __syncthreads();
    gpu::pdl_wait(); // launched while the kernel in front still runs
    for (int t = threadIdx.x; t < n; t += blockDim.x)
        route_token<E>(logits + (size_t)(t0 + t) * n_experts, n_experts, topk, idx + (size_t)(t0 + t) * topk,
                       wts + (size_t)(t0 + t) * topk, [&](int s, int e) {
                           ticket[t * topk + s] = (unsigned short)atomicAdd(&count[e], 1u);
                           expert[t * topk + s] = (unsigned char)e;
                       });
    __syncthreads();
    if constexpr (C > 1) {
        sm100::cluster_wait();
        for (int i = threadIdx.x; i < C * n_experts; i += blockDim.x) {
            const int to = i / n_experts, e = i - to * n_experts;
            sm100::st_cluster_u32(sm100::map_to_cta(sm100::smem_u32(&all[me][e]), to), count[e]);
        }
        sm100::cluster_sync_all(); // nobody touches another block's memory after this
    }
    if (threadIdx.x < 32) {
        // experts in front of expert e, then the blocks in front of this one
        unsigned before = 0;
#pragma unroll
        for (int h = 0; h < ROUTE_MAX_EXPERTS; h += 32) {
            const int e = h + lane;
            unsigned total = 0, mine = 0;
            if (e < n_experts) {
#pragma unroll
                for (int c = 0; c < C; c++) {
                    const unsigned v = C > 1 ? all[c][e] : count[e];
                    mine += c < me ? v : 0;
                    total += v;
                }
                if (me == 0)
                    counts[e] = total;
            }
            unsigned sum = total;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned up = __shfl_up_sync(0xffffffffu, sum, o);
                sum += lane >= o ? up : 0;
            }
            if (e < n_experts)
                offs[e] = before + sum - total + mine;
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n * topk; i += blockDim.x) {
        const unsigned p = offs[expert[i]] + ticket[i];
        order[p] = t0 * topk + i;
        pos[t0 * topk + i] = p;
    }
}

template <int E>
void launch_route(const float* logits, int n_tokens, int n_experts, int topk, long long* idx, float* wts, unsigned long long* counts,
                  long long* order, long long* pos, cudaStream_t st) {
    const bool wide = n_tokens >= ROUTE_CLUSTER_TOKENS;
    const int per = wide ? (n_tokens + ROUTE_CLUSTER - 1) / ROUTE_CLUSTER : n_tokens;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(wide ? ROUTE_CLUSTER : 1);
    cfg.blockDim = dim3(std::max(64, std::min(1024, (per + 31) / 32 * 32))); // a thread per token
    cfg.stream = st;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = ROUTE_CLUSTER;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = wide ? 2 : 1;
    CUDA_CHECK(cudaLaunchKernelEx(&cfg, wide ? route_one_launch_kernel<E, ROUTE_CLUSTER> : route_one_launch_kernel<E, 1>, logits, n_tokens,
                                  n_experts, topk, idx, wts, counts, order, pos));
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

// items (token, slot) up to which one launch does the whole routing: a block, or a cluster of eight
CCLX_API int cclx_moe_route_one_block() {
    return ROUTE_ONE_LAUNCH;
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
        if (n_tokens > 0 && (size_t)n_tokens * topk <= ROUTE_ONE_LAUNCH) {
            auto launch = n_experts <= 8 ? launch_route<8> : n_experts <= 16 ? launch_route<16> : launch_route<0>;
            launch(logits, n_tokens, n_experts, topk, idx, wts, (unsigned long long*)counts, order, pos, st);
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
    unsigned row, piece, pieces, step_rows, step_pieces;
    __device__ __forceinline__ piece_walk(unsigned warp, unsigned nwarps, unsigned n) : pieces(n) {
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

constexpr int MOE_THREADS = 512;

// A rank's tables in shared memory, read at once by all threads: followed pointer by pointer, their lines come one after the other through
// the caches in front of every barrier and address. Dispatch and combine of 8 emulated ranks together, K = 2: 62 tokens x 1112
// 83.8 -> 82.4 us, 1024 x 4096 127.3 -> 125.8; 2 ranks, 2048 x 4096 69.3 -> 68.4.
__device__ __forceinline__ void fetch_tables(const comm_dev* tab, const moe_args& a, comm_dev& c, moe_rank_args& ra) {
    const int er = a.emu ? (int)blockIdx.y : 0;
    static_assert(sizeof(comm_dev) % 8 == 0 && sizeof(moe_rank_args) % 8 == 0 && sizeof(comm_dev) / 8 <= MOE_THREADS / 2, "copied by words");
    const int i = threadIdx.x, j = threadIdx.x - MOE_THREADS / 2;
    if (i < (int)(sizeof(comm_dev) / 8))
        reinterpret_cast<unsigned long long*>(&c)[i] = reinterpret_cast<const unsigned long long*>(tab + er)[i];
    if (a.emu && j >= 0 && j < (int)(sizeof(moe_rank_args) / 8))
        reinterpret_cast<unsigned long long*>(&ra)[j] = reinterpret_cast<const unsigned long long*>(a.emu_tab + er)[j];
    if (!a.emu && j == 0)
        ra = a.r0;
    __syncthreads();
}
constexpr int MOE_SEGMENTS = 256;

// Bound by memory (every row read once, written topk times).  The rows stand grouped by expert, but are not sent in that order:
// each expert's rows are cut into the same number of parts and the parts are taken in turn, so that all peers receive all the time,
// and the topk copies of a token, which is found at about the same depth of every list, are read while it is still in the L2.
// The table of parts is made while the barrier's flags travel: in front of it, it cost an exchange of few rows what the order gains.
// Eight ranks on one GPU, top-2, each launch by itself: 1024 tokens of 4096 47.7 us in order of experts with one piece per warp in
// flight, 42.8 with the table in front of the barrier, 41.0 now; 256 of 4096 21.8, 22.9 and 21.7; 62 of 1112 16.2, 16.5 and 15.3; one of
// 512 15.5, 15.4 and 14.5, the barriers alone.
__global__ void __launch_bounds__(MOE_THREADS) moe_dispatch_kernel(const comm_dev* tab, moe_args a) {
    __shared__ comm_dev c;
    __shared__ moe_rank_args ra;
    fetch_tables(tab, a, c, ra);
    block_sync s;
    sync_begin(c, s);
    const int W = c.world;
    __shared__ int s_cnt[MAX_RANKS * MAX_RANKS], s_own[MAX_RANKS], s_dst[MAX_RANKS], s_pre[MAX_RANKS + 1], s_over;
    __shared__ unsigned s_seg[MOE_SEGMENTS]; // number of rows taken before segment part * W + expert
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
    peer_arrive(c, s);
    const int shift = 31 - __clz(MOE_SEGMENTS / W), n_seg = W << shift; // 2^shift parts
    auto upto = [&](int e, int part) { return (unsigned)(((unsigned long long)(unsigned)s_own[e] * (unsigned)part) >> shift); };
    for (int i = threadIdx.x; i < MOE_SEGMENTS; i += blockDim.x) {
        const int part = i / W, e = i % W;
        unsigned n = 0;
        if (i < n_seg)
            for (int q = 0; q < W; q++)
                n += upto(q, q < e ? part + 1 : part);
        s_seg[i] = i < n_seg ? n : 0xffffffffu;
    }
    if (threadIdx.x <= W) {
        int pre = 0;
        for (int q = 0; q < (int)threadIdx.x; q++)
            pre += s_own[q];
        s_pre[threadIdx.x] = pre;
    }
    if (threadIdx.x == 0)
        s_over = 0;
    __syncthreads();

    // A warp moves up to 256 packs of a row at a time, eight per lane, reads the next ones before it writes these, and fetches the
    // index of the row after that meanwhile; its first piece is on its way during the barrier.  Pieces instead of rows: 2048 rows
    // among 288 warps are 8 rounds for 7.1 rows each, their halves 15 for 14.2 (the last barrier waited 8 us for the slowest of 50).
    struct piece {
        const uint4* src; // null: none left
        int first; // pack of this lane
        int e; // owner of the expert
        unsigned j; // place among the rows this rank sends there
    };
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5, packs = a.hidden / 8;
    piece_walk w(blockIdx.x * wpb + (threadIdx.x >> 5), gridDim.x * wpb, (packs + 255) / 256);
    const unsigned rows = (unsigned)s_pre[W], n_items = (unsigned)a.n_items;
    int next_e = 0, next_item = -1;
    unsigned next_j = 0;
    auto look = [&] { // for the row that the walk has come to
        if (w.row >= rows)
            return;
        int seg = 0;
#pragma unroll
        for (int k = 0; k < MOE_SEGMENTS / 32; k++)
            seg += s_seg[lane + 32 * k] <= w.row;
        seg = __reduce_add_sync(0xffffffffu, seg) - 1;
        const int part = seg / W;
        next_e = seg - part * W;
        next_j = upto(next_e, part) + (w.row - s_seg[seg]);
        const unsigned i = (unsigned)s_pre[next_e] + next_j;
        next_item = i < n_items ? (int)ra.order[i] : -1; // counts that promise more rows than there are
    };
    auto fetch = [&](piece& p, uint4 (&v)[8]) {
        p.src = nullptr;
        if (w.row >= rows)
            return;
        p.e = next_e;
        p.j = next_j;
        p.first = next_item < 0 ? packs : (int)w.piece * 256 + lane;
        p.src = reinterpret_cast<const uint4*>(ra.x + (size_t)((unsigned)max(next_item, 0) / (unsigned)a.topk) * a.hidden);
        w.next();
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (p.first + k * 32 < packs)
                v[k] = p.src[p.first + k * 32];
        look();
    };
    auto put = [&](const piece& p, const uint4 (&v)[8]) {
        char* dst = c.heap[p.e] + a.buf_off + ((size_t)(unsigned)s_dst[p.e] + p.j) * (size_t)a.hidden * 2;
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (p.first + k * 32 < packs)
                st16(dst + (size_t)(p.first + k * 32) * 16, v[k]);
    };
    piece p0, p1;
    uint4 v0[8], v1[8];
    look();
    fetch(p0, v0);

    const bool ok = peer_wait(c, s);
    // The table is read by all threads at once and worked on in shared memory: one thread that walked it in global memory
    // waited W * W times for the L2, some 40 us for eight ranks, in every block.
    for (int i = threadIdx.x; i < W * W; i += blockDim.x)
        s_cnt[i] = __ldcv(reinterpret_cast<const int*>(c.heap[c.rank] + a.cnt_off) + blk_words + i);
    __syncthreads();
    if (threadIdx.x < W) {
        const int e = threadIdx.x;
        int off = 0, tot = 0;
        for (int q = 0; q < W; q++) {
            const int v = s_cnt[q * W + e];
            off += q < c.rank ? v : 0;
            tot += v;
        }
        s_dst[e] = off;
        if (tot > (long long)a.cap_rows)
            s_over = 1;
        if (blockIdx.x == 0) {
            ra.meta[e] = off;
            ra.meta[W + e] = s_pre[e];
            if (e == c.rank)
                ra.meta[2 * W] = tot;
        }
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0)
        ra.meta[2 * W + 1] = s_over;
    if (ok && !s_over) {
        while (p0.src) {
            fetch(p1, v1);
            put(p0, v0);
            if (!p1.src)
                break;
            fetch(p0, v0);
            put(p1, v1);
        }
    }
    peer_barrier(c, s);
    sync_end(c, s, gridDim.x, 2, false);
}

// Bound by memory (topk rows read for every row written).  A warp works on one token at a time: lane sl finds out where the row
// of slot sl lies (expert, place, weight: three dependent loads) for the warp's next token while the rows of this one are summed.
// TOPK 1 and 2 keep 16 packs per lane in flight and finish a pack at once (the case above: 47.8 us with 8 and sums that wait
// for all slots, now 43.4); 0, any number of slots, two packs of two slots.
template <int TOPK>
__global__ void __launch_bounds__(MOE_THREADS) moe_combine_kernel(const comm_dev* tab, moe_args a) {
    __shared__ comm_dev c;
    __shared__ moe_rank_args ra;
    fetch_tables(tab, a, c, ra);
    block_sync s;
    sync_begin(c, s);
    const int W = c.world;
    // every owner has finished its expert FFN (this launch is ordered after it on each rank's stream)
    bool ok = peer_barrier(c, s);
    if (ok) {
        const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
        const unsigned warp = blockIdx.x * wpb + (threadIdx.x >> 5), nwarps = gridDim.x * wpb;
        const int packs = a.hidden / 8, topk = TOPK ? TOPK : a.topk;
        const unsigned tokens = (unsigned)(a.n_items / (unsigned)topk);
        auto locate = [&](unsigned t, int sl0, const char*& row, float& w) {
            row = nullptr;
            w = 0.f;
            if (t < tokens && sl0 + lane < topk) {
                const size_t f = (size_t)t * topk + sl0 + lane;
                const int e = (int)ra.expert[f];
                const long long p = ra.pos[f];
                w = ra.weight[f];
                row = c.heap[e] + a.buf_off + (size_t)(ra.meta[e] + (p - ra.meta[W + e])) * (size_t)a.hidden * 2;
            }
        };
        auto add = [&](float w, const uint4& u, float (&acc)[8]) {
            const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(&u);
#pragma unroll
            for (int q = 0; q < 8; q++)
                acc[q] = fmaf(w, __bfloat162float(b[q]), acc[q]);
        };
        auto store = [&](unsigned t, int k, const float (&acc)[8]) {
            uint4 o;
            __nv_bfloat16* oh = reinterpret_cast<__nv_bfloat16*>(&o);
#pragma unroll
            for (int q = 0; q < 8; q++)
                oh[q] = __float2bfloat16_rn(acc[q]);
            reinterpret_cast<uint4*>(ra.out + (size_t)t * a.hidden)[k] = o;
        };
        const char* next_row;
        float next_w;
        locate(warp, 0, next_row, next_w);
        for (unsigned t = warp; t < tokens; t += nwarps) {
            const char* my_row = next_row;
            float my_w = next_w;
            locate(t + nwarps, 0, next_row, next_w);
            if constexpr (TOPK > 0) {
                constexpr int U = 16 / TOPK;
                const char* row[TOPK];
                float w[TOPK];
#pragma unroll
                for (int h = 0; h < TOPK; h++) {
                    row[h] = (const char*)__shfl_sync(0xffffffffu, (unsigned long long)my_row, h);
                    w[h] = __shfl_sync(0xffffffffu, my_w, h);
                }
                for (int k0 = lane; k0 < packs; k0 += 32 * U) {
                    uint4 v[TOPK][U];
#pragma unroll
                    for (int h = 0; h < TOPK; h++)
#pragma unroll
                        for (int k = 0; k < U; k++)
                            if (k0 + k * 32 < packs)
                                v[h][k] = ld_cv16(row[h] + (size_t)(k0 + k * 32) * 16);
#pragma unroll
                    for (int k = 0; k < U; k++)
                        if (k0 + k * 32 < packs) {
                            float acc[8] = {};
#pragma unroll
                            for (int h = 0; h < TOPK; h++)
                                add(w[h], v[h][k], acc);
                            store(t, k0 + k * 32, acc);
                        }
                }
            }
            else {
                for (int k0 = lane; k0 < (packs + 31) / 32 * 32; k0 += 64) {
                    float acc[2][8] = {};
                    for (int sl = 0; sl < topk; sl += 2) {
                        if (topk > 32 && sl % 32 == 0) // more slots than lanes
                            locate(t, sl, my_row, my_w);
                        uint4 v[2][2];
                        float w[2];
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int from = min(sl + h, topk - 1) & 31;
                            const char* row = (const char*)__shfl_sync(0xffffffffu, (unsigned long long)my_row, from);
                            w[h] = __shfl_sync(0xffffffffu, my_w, from);
                            if (sl + h < topk)
#pragma unroll
                                for (int k = 0; k < 2; k++)
                                    if (k0 + k * 32 < packs)
                                        v[h][k] = ld_cv16(row + (size_t)(k0 + k * 32) * 16);
                        }
#pragma unroll
                        for (int h = 0; h < 2; h++)
                            if (sl + h < topk)
#pragma unroll
                                for (int k = 0; k < 2; k++)
                                    if (k0 + k * 32 < packs)
                                        add(w[h], v[h][k], acc[k]);
                    }
#pragma unroll
                    for (int k = 0; k < 2; k++)
                        if (k0 + k * 32 < packs)
                            store(t, k0 + k * 32, acc[k]);
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
    auto kernel = dispatch ? moe_dispatch_kernel
                  : a.topk == 1 ? moe_combine_kernel<1>
                  : a.topk == 2 ? moe_combine_kernel<2>
                                : moe_combine_kernel<0>;
    if (dc.emulated()) {
        static_assert(sizeof(moe_rank_args) <= sizeof(dev::rank_args), "argument block too large");
        a.emu = 1;
        a.emu_tab = (const moe_rank_args*)dc.emu_table(dispatch ? gpu::device_comm::EMU_DISPATCH : gpu::device_comm::EMU_COMBINE, ra,
                                                       dc.world() * sizeof(moe_rank_args), st);
        const comm_dev* tab = dc.table();
        void* argv[] = { (void*)&tab, (void*)&a };
        dim3 grid(blocks, dc.world());
        CUDA_CHECK(cudaLaunchCooperativeKernel((const void*)kernel, grid, dim3(MOE_THREADS), argv, 0, st));
    }
    else {
        a.emu = 0;
        a.emu_tab = nullptr;
        kernel<<<blocks, MOE_THREADS, 0, st>>>(dc.table(), a);
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
