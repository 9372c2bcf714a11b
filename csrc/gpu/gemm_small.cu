// bf16 GEMM for products that leave the CTA-pair kernel's 256 x 256 tiles without enough of them: few rows of A
// (decoding, a lightly loaded expert), or a small C.  C[M,N] = act(A[M,K] * B[N,K]^T), fp32 accumulation.
//
// The operands change places: 128 rows of B are the M side of tcgen05.mma and TN = 16 ... 128 rows of A its N side, so
// two dozen tokens cost 32 columns, not 128 rows of which most are padding.  K is cut over the S CTAs of a cluster;
// each reads its own part of B once and accumulates in its tensor memory, then every CTA of the cluster adds up
// TN / S columns from the partial sums the others stored into its shared memory (fixed order, fp32), applies the
// activation and writes bf16.  No workspace, no second kernel, no atomics.
//
// What bounds it: with few rows the bytes of B, with few tiles the time of a step.  K is cut 1 to 8 times, in whatever way fills the
// SMs once (1 x 1272 x 11552: 18.0 us on 40 CTAs, 11.2 on 80; 512 x 1024 x 4096: 15.5 us with 4 x 128 columns, 11.8 with 4 x 64).  A
// ring takes half of an SM's shared memory, 24 x 14336 x 4096: 117 MB in 23.6 us = 5.0 TB/s; only tiles of 128 rows that are
// alone on their SM gain from the whole of it (73 x 5632 x 10232, K cut in 3: 42.7 us, now 29.1).  The next kernel is not let in
// early: its CTAs took the room that this one's clusters need (a call after another 6 % slower).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <iterator>

#include "core/env.hpp"
#include "core/log.hpp"
#include "gpu/cuda_driver.hpp"
#include "gpu/fused_gemm.cuh"
#include "gpu/fused_gemm.hpp"
#include "gpu/launch_util.cuh"

namespace cclx {
namespace gpu {

namespace {

constexpr int GS_BN = 128; // rows of B per tile

struct gemm_small_params {
    CUtensorMap tmA; // [M,K], box 64 x TN
    CUtensorMap tmB; // [N,K], box 64 x 128
    __nv_bfloat16* C;
    uint32_t* err;
    int M, N, K, epilogue;
    int splits; // CTAs per cluster: 1 to 8
    uint32_t inv_splits; // 65536 / splits, rounded up
    int pitch; // units of four columns that a CTA finishes, at most
    unsigned long long timeout_ns;
    const int* rows; // optional device word: only the first min(M, *rows) rows of A are multiplied
};

// Stages of the ring are a constant of the kernel: with a number known at launch alone the loops took 0.3 us of a 6 us product
// longer.  Four leave room for two CTAs per SM; more of them slow the loads from memory down (2 x 6176 x 5432: 15.7 us with 4,
// 16.2 with 6), but for 128 rows, where a CTA that is alone on its SM takes the whole of it.
constexpr int GS_STAGES_ALONE = 6;

template <int TN, int STAGES>
struct gs_layout {
    static constexpr int B_STAGE = GS_BN * GEMM_BK * 2;
    static constexpr int A_STAGE = TN * GEMM_BK * 2;
    static constexpr int STAGE = A_STAGE + B_STAGE;
    static constexpr int TMEM_COLS = TN < 32 ? 32 : TN;
    static constexpr int BLOCKS = STAGES > 4 ? 1 : 2; // per SM
    static constexpr int UNITS = TN / 4; // of four columns: what the CTAs of a cluster share out
    // of four epilogue warps, a share of the columns each: 200 x 1752 x 11840 took 22.8 us with one of them, 313 x 1720 x 864 7.3,
    // now 20.8 and 6.8
    static constexpr int GROUPS = TN >= 64 ? 2 : 1;
    static constexpr int THREADS = 64 + 128 * GROUPS;
    static constexpr int TOTAL = 1024 + STAGES * STAGE + 128;
    // the ring also holds the partial sums afterwards: a source's units for one CTA, rounded up, times up to 8 sources
    static_assert((UNITS + 7) * GS_BN * 16 <= STAGES * STAGE, "the partial sums must fit the ring");
};

__device__ __forceinline__ void gs_fail(const gemm_small_params& P, volatile int* abort_flag, uint32_t detail) {
    *abort_flag = 1;
    if (P.err && P.err[0] == GE_OK) {
        P.err[1] = blockIdx.x;
        P.err[2] = detail;
        __threadfence();
        P.err[0] = GE_MBAR_TIMEOUT;
    }
}

// four columns (rows tok ... tok + 3 of A) of row n0 + row of B: activation, then neighbouring lanes swap halves and
// write pairs, the even lane columns 0 and 1, the odd lane columns 2 and 3.  Whole warps.
__device__ __forceinline__ void gs_store(const gemm_small_params& P, int M, int tok, int n0, int row, const float (&x)[4]) {
    float v[4] = { x[0], x[1], x[2], x[3] };
    if (P.epilogue == EPI_SILU) {
#pragma unroll
        for (int k = 0; k < 4; k++)
            v[k] = silu_f(v[k]);
    }
    const bool odd = row & 1;
    const float g0 = __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[2], 1);
    const float g1 = __shfl_xor_sync(0xffffffffu, odd ? v[1] : v[3], 1);
    const float k0 = odd ? v[2] : v[0], k1 = odd ? v[3] : v[1];
    tok += odd ? 2 : 0;
    const int n = n0 + (row & ~1);
    __nv_bfloat16* dst = P.C + (size_t)tok * P.N + n;
    if (n < P.N && tok < M)
        *reinterpret_cast<__nv_bfloat162*>(dst) = odd ? __floats2bfloat162_rn(g0, k0) : __floats2bfloat162_rn(k0, g0);
    if (n < P.N && tok + 1 < M)
        *reinterpret_cast<__nv_bfloat162*>(dst + P.N) = odd ? __floats2bfloat162_rn(g1, k1) : __floats2bfloat162_rn(k1, g1);
}

// adds the S partial sums of every GROUPS-th of this CTA's units of four columns, from `first` on, in order and stores the result;
// one thread of a group per row of B
template <int GROUPS>
__device__ __forceinline__ void gs_reduce(const gemm_small_params& P, int S, int M, uint32_t part, int pitch, int first, int units,
                                          int tok, int n0, int row) {
    const uint32_t step = (uint32_t)pitch * GS_BN * 16;
    part += first * GS_BN * 16;
    for (int u = first; u < units && tok + 4 * u < M; u += GROUPS, part += GROUPS * GS_BN * 16) {
        float v[8][4];
#pragma unroll
        for (int s = 0; s < 8; s++)
            if (s < S)
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v[s][0]), "=f"(v[s][1]), "=f"(v[s][2]), "=f"(v[s][3])
                             : "r"(part + s * step));
#pragma unroll
        for (int s = 1; s < 8; s++)
            if (s < S)
#pragma unroll
                for (int k = 0; k < 4; k++)
                    v[0][k] += v[s][k];
        gs_store(P, M, tok + 4 * u, n0, row, v[0]);
    }
}

template <int TN, int STAGES>
__global__ void __launch_bounds__(gs_layout<TN, STAGES>::THREADS, gs_layout<TN, STAGES>::BLOCKS)
    gemm_small_kernel(const __grid_constant__ gemm_small_params P) {
    using namespace sm100;
    typedef gs_layout<TN, STAGES> L;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sB = smem;
    uint8_t* sA = smem + STAGES * L::B_STAGE;
    uint64_t* bars = (uint64_t*)(smem + STAGES * L::STAGE);
    uint64_t* full = bars;
    uint64_t* empty = bars + STAGES;
    uint64_t* tfull = bars + 2 * STAGES;
    uint32_t* tmem_holder = (uint32_t*)(bars + 2 * STAGES + 1);
    volatile int* abort_flag = (volatile int*)(tmem_holder + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = P.splits, split = S > 1 ? (int)cluster_ctarank() : 0;
    const int n0 = (int)blockIdx.x / S * GS_BN, tok0 = (int)blockIdx.y * TN;
    const int KB = (P.K + GEMM_BK - 1) / GEMM_BK;
    const int kb0 = KB * split / S, kb1 = KB * (split + 1) / S;
    const unsigned long long limit = P.timeout_ns;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(tfull, 1);
        mbar_fence_init();
        tma_prefetch_desc(&P.tmA);
        tma_prefetch_desc(&P.tmB);
    }
    if (warp == 2) {
        tmem_alloc(tmem_holder, L::TMEM_COLS);
        tc_fence_before_sync();
    }
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_holder;
    pdl_wait(); // everything above overlaps the end of the kernel in front
    const int M = P.rows ? max(0, min(P.M, *P.rows)) : P.M;
    if (tok0 >= M) { // no rows: the same in all CTAs of the cluster
        if (warp == 2)
            tmem_dealloc(tmem, L::TMEM_COLS);
        return;
    }

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0, st = 0, ph = 0;
            for (int kb = kb0; kb < kb1; kb++, it++) {
                if (!mbar_wait(&empty[st], ph ^ 1, abort_flag, limit)) {
                    gs_fail(P, abort_flag, 2);
                    break;
                }
                mbar_expect_tx(&full[st], L::STAGE);
                tma_load_2d(sB + st * L::B_STAGE, &P.tmB, kb * GEMM_BK, n0, &full[st]);
                tma_load_2d(sA + st * L::A_STAGE, &P.tmA, kb * GEMM_BK, tok0, &full[st]);
                if (++st == STAGES) {
                    st = 0;
                    ph ^= 1;
                }
            }
            // copies still in flight land before the ring is used for anything else
            const uint32_t first = it > (uint32_t)STAGES ? it - STAGES : 0;
            for (uint32_t i = first; i < it; i++)
                mbar_wait(&full[i % STAGES], (i / STAGES) & 1, abort_flag, limit);
        }
        __syncwarp();
    }
    else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = make_idesc_bf16(GS_BN, TN);
            uint32_t st = 0, ph = 0;
            bool ok = true;
            for (int kb = kb0; kb < kb1; kb++) {
                if (!mbar_wait(&full[st], ph, abort_flag, limit)) {
                    gs_fail(P, abort_flag, 4);
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t b_addr = smem_u32(sB + st * L::B_STAGE), a_addr = smem_u32(sA + st * L::A_STAGE);
#pragma unroll
                for (int k = 0; k < GEMM_BK / GEMM_UMMA_K; k++)
                    umma_bf16(tmem, make_smem_desc_sw128(b_addr + k * GEMM_UMMA_K * 2),
                              make_smem_desc_sw128(a_addr + k * GEMM_UMMA_K * 2), idesc, (kb != kb0 || k != 0) ? 1u : 0u);
                umma_commit(&empty[st]);
                if (++st == STAGES) {
                    st = 0;
                    ph ^= 1;
                }
            }
            if (ok)
                umma_commit(tfull);
        }
        __syncwarp();
    }
    bool good = true;
    if (warp >= 2) {
        good = mbar_wait_warp(tfull, 0, abort_flag, limit);
        if (!good && lane == 0)
            gs_fail(P, abort_flag, 5);
        tc_fence_after_sync();
    }
    // every CTA of the cluster is done with its ring
    if (S > 1)
        cluster_sync_all();
    else
        __syncthreads();
    // The units of four columns are shared out among the cluster's CTAs: CTA s finishes units [UNITS s / S, UNITS (s + 1) / S).
    // Both numbers are small, so a multiplication divides by S exactly.
    auto first_unit = [&](uint32_t s) { return (uint32_t)L::UNITS * s * P.inv_splits >> 16; };
    const int pitch = P.pitch;
    const int q = warp & 3; // quarter of the tensor memory's lanes this warp may read
    const int grp = (warp - 2) >> 2, row = q * 32 + lane;
    constexpr int COLS = TN / L::GROUPS; // of this warp
    if (warp >= 2 && good) {
        // Partial sums travel as [source][unit][row] packs of four floats: a warp stores 512 contiguous bytes,
        // and the reader's lanes take consecutive rows.  An undivided K needs no exchange.
        const uint32_t base = smem_u32(smem) + (uint32_t)(split * pitch * GS_BN + row) * 16;
        uint32_t unit = grp * COLS / 4, owner = ((unit + 1) * S - 1) / L::UNITS, end = first_unit(owner + 1);
        uint32_t dst = S > 1 ? map_to_cta(base + (unit - first_unit(owner)) * GS_BN * 16, owner) : 0;
        constexpr int CH = COLS < 32 ? 16 : 32;
#pragma unroll 1
        for (int c0 = grp * COLS; c0 < (grp + 1) * COLS; c0 += CH) {
            uint32_t r[CH];
            if constexpr (CH == 16)
                tmem_ld_32x16(tmem + ((uint32_t)(q * 32) << 16) + c0, r);
            else
                tmem_ld_32x32(tmem + ((uint32_t)(q * 32) << 16) + c0, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < CH; i += 4) {
                if (S == 1) {
                    const float v[4] = { __uint_as_float(r[i]), __uint_as_float(r[i + 1]), __uint_as_float(r[i + 2]),
                                         __uint_as_float(r[i + 3]) };
                    gs_store(P, M, tok0 + c0 + i, n0, row, v);
                }
                else {
                    if (unit == end) {
                        owner++;
                        end = first_unit(owner + 1);
                        dst = map_to_cta(base, owner);
                    }
                    st_cluster_v4(dst, r[i], r[i + 1], r[i + 2], r[i + 3]);
                    dst += GS_BN * 16;
                    unit++;
                }
            }
        }
        tc_fence_before_sync();
    }
    if (S > 1)
        cluster_sync_all();
    else
        __syncthreads();
    if (S > 1 && warp >= 2 && !warp_sees(abort_flag)) {
        const uint32_t part = smem_u32(smem) + row * 16;
        const int u0 = first_unit(split), units = first_unit(split + 1) - u0, tok = tok0 + 4 * u0;
        gs_reduce<L::GROUPS>(P, S, M, part, pitch, grp, units, tok, n0, row);
    }
    if (warp == 2) { // all reads of the accumulator lie in front of the last barrier
        tc_fence_after_sync();
        tmem_dealloc(tmem, L::TMEM_COLS);
    }
}

// Stands for the kernels above when the runtime is asked how many clusters fit: for kernels with tensor memory it answers for one CTA
// per SM whatever shared memory allows, but two run (24 rows, K = 14336 in eight parts: 22.7 us for 4096 columns, 32 clusters, and
// 32.9 for 4352, 34 clusters where 33 fit in twos and 15 alone).
template <int TN, int STAGES>
__global__ void __launch_bounds__(gs_layout<TN, STAGES>::THREADS, gs_layout<TN, STAGES>::BLOCKS) gs_shape_kernel() {}

// Clusters of `splits` CTAs that run at the same time.  A cluster stays within a group of SMs, so there are fewer than SMs / splits with
// one CTA per SM, but more than twice as many with two: 15 and 33 clusters of eight, 33 and 71 of four.
template <int TN, int STAGES>
int resident_clusters(int dev, int splits) {
    typedef gs_layout<TN, STAGES> L;
    static std::atomic<int> known[64][9];
    if (splits == 1)
        return L::BLOCKS * device_sms();
    int n = dev < 64 ? known[dev][splits].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        allow_smem<gs_shape_kernel<TN, STAGES>>(L::TOTAL);
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(splits);
        cfg.blockDim = dim3(L::THREADS);
        cfg.dynamicSmemBytes = L::TOTAL;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = splits;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        CUDA_CHECK(cudaOccupancyMaxActiveClusters(&n, gs_shape_kernel<TN, STAGES>, &cfg));
        n = std::max(n, 1);
        if (dev < 64)
            known[dev][splits].store(n, std::memory_order_relaxed);
    }
    return n;
}
struct fits {
    int alone, in_twos;
};
fits clusters_that_fit(int dev, int splits) { // on the current device
    return { resident_clusters<128, GS_STAGES_ALONE>(dev, splits), resident_clusters<64, 4>(dev, splits) };
}

template <int TN, int STAGES>
void launch_small(const gemm_small_params& P, int tiles_n, int tiles_m, cudaStream_t st) {
    typedef gs_layout<TN, STAGES> L;
    allow_smem<gemm_small_kernel<TN, STAGES>>(L::TOTAL);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(tiles_n * P.splits, tiles_m);
    cfg.blockDim = dim3(L::THREADS);
    cfg.dynamicSmemBytes = L::TOTAL;
    cfg.stream = st;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = P.splits;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    CUDA_CHECK(cudaLaunchKernelEx(&cfg, gemm_small_kernel<TN, STAGES>, P));
}

// What a product costs with tiles of TN rows of A, in us: `fixed` from launch to output, `exchange` if K is cut, a step of 64
// of K with one CTA on an SM or with two, `crowd` once where some SM holds two, another round of resident CTAs, the factors on the
// steps where K is no multiple of 16, so that the rows of a box begin between the 32-byte sectors, and a round of CTAs that find no
// rows.  `drawn`: what a CTA that is alone on its SM draws from memory, in bytes per us; the ring limits that (64 x 14336 x
// 4096 on 112 CTAs of four stages 28.2 us, with K in two parts on 224 24.1).
//
// Fitted to 7800 times: 255 products of sizes that models have (1 to 2048 rows, N and K of 768 to 14336) and 380 drawn ones of 1 to
// 8000 rows, 500 to 14300 columns and K.  The chosen plan takes 0.7 % longer than the best one for the first, 1.0 % for the others,
// at most 1.2 times.  The fit before it, to drawn ones alone, took rows of tiles that run beside one another to read B once each
// and knew neither `crowd` nor `drawn`: 3.6 % and 1.5 %, at most 1.4 times (64 x 14336 x
// 4096 28.2 us, now 24.1; 128 x 2304 x 768 7.4 and 5.4; 192 x 4096 x 14336 45 and 39).
struct small_cost {
    int tn;
    double fixed, exchange, alone, two, crowd, round, ragged, ragged_two, idle, drawn;
};
constexpr small_cost SMALL_COSTS[] = {
    { 16, 2.64, 0.91, 0.245, 0.287, 0.63, 0.48, 1.21, 1.43, 0.31, 52e3 },
    { 32, 3.00, 0.83, 0.245, 0.308, 0.87, 2.45, 1.22, 1.43, 0.64, 52e3 },
    { 64, 3.20, 1.12, 0.244, 0.329, 1.40, 3.33, 1.31, 1.68, 0.69, 49e3 },
    { 128, 3.95, 1.71, 0.323, 0.455, 1.90, 5.35, 1.50, 1.65, 0.55, 39e3 },
};
constexpr small_cost SMALL_COST_ALONE = { 128, 3.95, 1.71, 0.251, 0, 0, 0, 1.50, 0, 0, 82e3 }; // GS_STAGES_ALONE
constexpr double SMALL_BYTES_PER_US = 6.5e6; // of B, from memory
constexpr double SMALL_L2_BYTES = 64e6; // of B that a later round of tiles still finds in the L2

// Expected time in us of `rows` of the M rows that the grid covers.
double small_us(const small_cost& cost, int s, const fits& clusters, int M, int rows, int N, int K) {
    const int kb = (K + GEMM_BK - 1) / GEMM_BK, across = (N + GS_BN - 1) / GS_BN, down = (rows + cost.tn - 1) / cost.tn;
    const long long tiles = (long long)across * down, launched = (long long)across * ((M + cost.tn - 1) / cost.tn);
    const long long one = clusters.alone, most = clusters.in_twos; // at the same time
    const small_cost& c = cost.tn == SMALL_COST_ALONE.tn && launched <= one ? SMALL_COST_ALONE : cost;
    const long long rounds = (tiles + most - 1) / most, idle = (launched + most - 1) / most - rounds;
    const bool alone = tiles <= one;
    double steps = (double)rounds * ((kb + s - 1) / s) * (alone ? c.alone : c.two);
    if (K % 16)
        steps *= alone ? c.ragged : c.ragged_two;
    double bytes = (double)N * K * 2, rate = SMALL_BYTES_PER_US;
    if (bytes > SMALL_L2_BYTES) {
        // rows of tiles that run beside one another read B from memory once, but do not keep step to the end
        const double reads = (double)std::min<long long>(down, rounds);
        bytes *= reads + 0.1 * (down - reads);
        if (alone)
            rate = std::min(rate, c.drawn * (double)(tiles * s));
    }
    // both limits are felt where they are close: the fourth root of the sum of the fourth powers
    const double stream = bytes / rate, s2 = steps * steps, m2 = stream * stream;
    return c.fixed + (s > 1 ? c.exchange : 0) + std::sqrt(std::sqrt(s2 * s2 + m2 * m2)) + (alone ? 0 : c.crowd) +
           c.round * (rounds - 1) + c.idle * idle;
}

} // namespace

// Up to 128 rows this kernel, beyond that by the estimates.  The line this draws at 4096 x 4096 lies between 256 rows (17.2 us here,
// 18.5 with pairs) and 512 (22.6 and 19.1), at 1024 x 4096 between 1024 rows (16.2 and 17.8) and 2048 (21.9 and 18.8).
//
// A row count that only the device knows is M at most, and what it is depends on the caller (a layer that gathers from W ranks: M / W).
// The plan is the one that loses least in the worst of M / 8, M / 4, M / 2 and M rows, measured by the best plan of each.  Over 79
// products of five counts each its times are 5.0 % above the best plans'; with the best plan of M / 2 7.5 %, and then up to 1.7 times
// where B is read again for a second row of tiles (92 x 12680 x 11464, all rows: 109 us, now 76; 99 x 10664 x 6136: 62 and 38);
// with the best plan of M 8.5 %.
//
// The answer depends on the sizes and the kind of device alone and takes 0.5 us to work out, 2 us where the count is on the device, of
// the 4.2 us of a call: each thread keeps its latest ones.
static gemm_choice choose_by_sizes(int M, int N, int K, bool rows_on_device) {
    CCL_THROW_IF_NOT(M > 0 && N > 0 && K > 0 && N % 8 == 0 && K % 8 == 0, "unsupported GEMM shape ", M, "x", N, "x", K);
    struct entry {
        int dev = -1, M, N, K;
        bool rows;
        gemm_choice c;
    };
    static thread_local entry known[64];
    int dev = 0;
    CUDA_CHECK(cudaGetDevice(&dev));
    entry& e = known[((unsigned)M * 31 + (unsigned)N * 17 + (unsigned)K * 5 + rows_on_device) / 8 % 64];
    if (e.dev == dev && e.M == M && e.N == N && e.K == K && e.rows == rows_on_device)
        return e.c;

    struct plan {
        int tn, splits, pairs; // pairs > 0: that kernel
        double us[4];
    } plans[8 * std::size(SMALL_COSTS) + 2];
    int n = 0;
    const int counts = rows_on_device ? 4 : 1;
    double best[4] = { 1e30, 1e30, 1e30, 1e30 };
    auto consider = [&](int tn, int splits, int pairs, auto&& us) {
        plan& p = plans[n++] = { tn, splits, pairs, {} };
        for (int i = 0; i < counts; i++) {
            p.us[i] = us((int)(((long long)M + (1 << i) - 1) >> i)); // M, M / 2, M / 4, M / 8
            best[i] = std::min(best[i], p.us[i]);
        }
    };
    const int kb = (K + GEMM_BK - 1) / GEMM_BK, across = (N + GS_BN - 1) / GS_BN;
    fits clusters[9];
    for (int s = 1; s <= 8; s++)
        clusters[s] = clusters_that_fit(dev, s);
    for (const small_cost& c : SMALL_COSTS) {
        if (c.tn >= 4 * std::max(M, 16)) // mostly padding
            break;
        for (int s = 1; s <= std::min(8, c.tn / 4) && (s == 1 || kb / s >= 2); s++) {
            // a second round of wide clusters waits for whole groups of SMs
            if (s > 2 && (long long)across * ((M + c.tn - 1) / c.tn) > clusters[s].in_twos)
                break;
            consider(c.tn, s, 0, [&](int rows) { return small_us(c, s, clusters[s], M, rows, N, K); });
        }
    }
    if (M > 128)
        for (int pairs = 1; pairs <= 2; pairs++)
            consider(0, 0, pairs, [&](int rows) { return gemm_2sm_estimate(rows, N, K, pairs); });

    gemm_choice c{ true, 0, 0, gemm_2sm_estimate(M, N, K, 2) < gemm_2sm_estimate(M, N, K, 1) ? 2 : 1 };
    double small = 1e30, pairs = 1e30;
    for (int i = 0; i < n; i++) {
        double worst = 0;
        for (int k = 0; k < counts; k++)
            worst = std::max(worst, plans[i].us[k] / best[k]);
        double& least = plans[i].pairs ? pairs : small;
        if (worst >= least)
            continue;
        least = worst;
        if (plans[i].pairs)
            c.pairs = plans[i].pairs;
        else {
            c.tn = plans[i].tn;
            c.splits = plans[i].splits;
        }
    }
    c.small = small < pairs;
    e = { dev, M, N, K, rows_on_device, c };
    return c;
}

// This kernel stores pairs of columns, the others packs of eight: an output between 16-byte boundaries is its own.
gemm_choice choose_gemm(const void* C, int M, int N, int K, bool rows_on_device) {
    gemm_choice c = choose_by_sizes(M, N, K, rows_on_device);
    CCL_THROW_IF_NOT(((uintptr_t)C & 3) == 0, "GEMM output must be 4-byte aligned");
    c.small |= ((uintptr_t)C & 15) != 0;
    return c;
}

void gemm_bf16_small(const void* A, const void* B, void* C, int M, int N, int K, int epilogue, uint32_t* err, cudaStream_t st,
                     const int* rows_dev, const gemm_choice& plan) {
    CCL_THROW_IF_NOT(M > 0 && N > 0 && K > 0 && N % 8 == 0 && K % 8 == 0, "unsupported GEMM shape ", M, "x", N, "x", K);
    gemm_small_params P;
    std::memset(&P, 0, sizeof(P));
    P.tmA = make_bf16_map(A, M, K, plan.tn);
    P.tmB = make_bf16_map(B, N, K, GS_BN);
    P.C = (__nv_bfloat16*)C;
    P.err = err;
    P.M = M;
    P.N = N;
    P.K = K;
    P.epilogue = epilogue;
    P.splits = plan.splits;
    P.inv_splits = (65536u + plan.splits - 1) / plan.splits;
    P.pitch = (plan.tn / 4 + plan.splits - 1) / plan.splits;
    P.rows = rows_dev;
    P.timeout_ns = (unsigned long long)env_data::get().wait_timeout_ms * 1000000ull;
    const int tiles_n = (N + GS_BN - 1) / GS_BN, tiles_m = (M + plan.tn - 1) / plan.tn;
    switch (plan.tn) {
        case 16: launch_small<16, 4>(P, tiles_n, tiles_m, st); break;
        case 32: launch_small<32, 4>(P, tiles_n, tiles_m, st); break;
        case 64: launch_small<64, 4>(P, tiles_n, tiles_m, st); break;
        default: {
            int dev = 0;
            CUDA_CHECK(cudaGetDevice(&dev));
            if ((long long)tiles_n * tiles_m <= clusters_that_fit(dev, plan.splits).alone)
                launch_small<128, GS_STAGES_ALONE>(P, tiles_n, tiles_m, st);
            else
                launch_small<128, 3>(P, tiles_n, tiles_m, st);
        }
    }
}

} // namespace gpu
} // namespace cclx
