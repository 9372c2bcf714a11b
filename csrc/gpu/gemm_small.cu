// bf16 GEMM for products that leave the CTA-pair kernel's 256 x 256 tiles without enough of them: few rows of A
// (decoding, a lightly loaded expert), or a small C.  C[M,N] = act(A[M,K] * B[N,K]^T), fp32 accumulation.
//
// The operands change places: 128 rows of B are the M side of tcgen05.mma and TN = 16 ... 256 rows of A its N side, so
// two dozen tokens cost 32 columns, not 128 rows of which most are padding.  K is cut over the S CTAs of a cluster;
// each reads its own part of B once and accumulates in its tensor memory, then every CTA of the cluster adds up
// TN / S columns from the partial sums the others stored into its shared memory (fixed order, fp32), applies the
// activation and writes bf16.  No workspace, no second kernel, no atomics.
//
// What bounds it: with few rows the bytes of B.  Two CTAs per SM with 72 to 96 KB of loads in flight each are more than
// the memory needs (24 x 14336 x 4096: 117 MB in 23.8 us = 4.9 TB/s; one 128 x 256 tile per CTA on 56 of 148 SMs
// took 81 us).
#include <algorithm>
#include <cstring>

#include "core/env.hpp"
#include "core/log.hpp"
#include "gpu/cuda_driver.hpp"
#include "gpu/fused_gemm.cuh"
#include "gpu/fused_gemm.hpp"
#include "gpu/launch_util.cuh"

namespace cclx {
namespace gpu {

CUtensorMap make_bf16_kmajor_map(const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows);

namespace {

constexpr int GS_BN = 128; // rows of B per tile

struct gemm_small_params {
    CUtensorMap tmA; // [M,K], box 64 x TN
    CUtensorMap tmB; // [N,K], box 64 x 128
    __nv_bfloat16* C;
    uint32_t* err;
    int M, N, K, epilogue;
    int splits; // CTAs per cluster: 1, 2, 4 or 8
    unsigned long long timeout_ns;
    const int* rows; // optional device word: only the first min(M, *rows) rows of A are multiplied
};

template <int TN>
struct gs_layout {
    static constexpr int STAGES = TN == 128 ? 3 : 4;
    static constexpr int B_STAGE = GS_BN * GEMM_BK * 2;
    static constexpr int A_STAGE = TN * GEMM_BK * 2;
    static constexpr int RING = STAGES * (A_STAGE + B_STAGE); // also holds the 128 x TN partial sums afterwards
    static constexpr int TOTAL = 1024 + RING + 128;
    static constexpr int TMEM_COLS = TN < 32 ? 32 : TN;
    static constexpr int BLOCKS = TN == 256 ? 1 : 2; // per SM
    static_assert(GS_BN * TN * 4 <= RING, "the partial sums must fit the ring");
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

// adds the S partial sums of this CTA's columns in order and stores the result; one thread per row of B
template <int S>
__device__ __forceinline__ void gs_reduce(const gemm_small_params& P, int M, uint32_t part, int cols, int tok, int n0, int row) {
#pragma unroll 2
    for (int c = 0; c < cols && tok + c < M; c += 4) {
        float v[S][4];
#pragma unroll
        for (int s = 0; s < S; s++)
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                         : "=f"(v[s][0]), "=f"(v[s][1]), "=f"(v[s][2]), "=f"(v[s][3])
                         : "r"(part + (uint32_t)(s * cols + c) * GS_BN * 4));
#pragma unroll
        for (int s = 1; s < S; s++)
#pragma unroll
            for (int k = 0; k < 4; k++)
                v[0][k] += v[s][k];
        gs_store(P, M, tok + c, n0, row, v[0]);
    }
}

template <int TN>
__global__ void __launch_bounds__(GEMM_THREADS, gs_layout<TN>::BLOCKS)
    gemm_small_kernel(const __grid_constant__ gemm_small_params P) {
    using namespace sm100;
    typedef gs_layout<TN> L;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sB = smem;
    uint8_t* sA = smem + L::STAGES * L::B_STAGE;
    uint64_t* bars = (uint64_t*)(smem + L::RING);
    uint64_t* full = bars;
    uint64_t* empty = bars + L::STAGES;
    uint64_t* tfull = bars + 2 * L::STAGES;
    uint32_t* tmem_holder = (uint32_t*)(bars + 2 * L::STAGES + 1);
    volatile int* abort_flag = (volatile int*)(tmem_holder + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = P.splits, split = S > 1 ? (int)cluster_ctarank() : 0;
    const int n0 = (int)blockIdx.x / S * GS_BN, tok0 = (int)blockIdx.y * TN;
    const int KB = (P.K + GEMM_BK - 1) / GEMM_BK;
    const int kb0 = KB * split / S, kb1 = KB * (split + 1) / S;
    const unsigned long long limit = P.timeout_ns;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < L::STAGES; i++) {
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
    const bool live = tok0 < M; // the same in all CTAs of the cluster

    if (warp == 0 && live) {
        if (lane == 0) {
            uint32_t it = 0;
            for (int kb = kb0; kb < kb1; kb++, it++) {
                const uint32_t st = it % L::STAGES, ph = (it / L::STAGES) & 1;
                if (!mbar_wait(&empty[st], ph ^ 1, abort_flag, limit)) {
                    gs_fail(P, abort_flag, 2);
                    break;
                }
                mbar_expect_tx(&full[st], L::A_STAGE + L::B_STAGE);
                tma_load_2d(sB + st * L::B_STAGE, &P.tmB, kb * GEMM_BK, n0, &full[st]);
                tma_load_2d(sA + st * L::A_STAGE, &P.tmA, kb * GEMM_BK, tok0, &full[st]);
            }
            // copies still in flight land before the ring is used for anything else
            const uint32_t first = it > (uint32_t)L::STAGES ? it - L::STAGES : 0;
            for (uint32_t i = first; i < it; i++)
                mbar_wait(&full[i % L::STAGES], (i / L::STAGES) & 1, abort_flag, limit);
        }
        __syncwarp();
    }
    else if (warp == 1 && live) {
        if (lane == 0) {
            constexpr uint32_t idesc = make_idesc_bf16(GS_BN, TN);
            uint32_t it = 0;
            bool ok = true;
            for (int kb = kb0; kb < kb1; kb++, it++) {
                const uint32_t st = it % L::STAGES, ph = (it / L::STAGES) & 1;
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
                              make_smem_desc_sw128(a_addr + k * GEMM_UMMA_K * 2), idesc, (it | k) != 0 ? 1u : 0u);
                umma_commit(&empty[st]);
            }
            if (ok)
                umma_commit(tfull);
        }
        __syncwarp();
    }
    bool good = live;
    if (warp >= 2 && live) {
        good = mbar_wait(tfull, 0, abort_flag, limit);
        if (!good && lane == 0)
            gs_fail(P, abort_flag, 5);
        tc_fence_after_sync();
    }
    // every CTA of the cluster is done with its ring
    if (S > 1)
        cluster_sync_all();
    else
        __syncthreads();
    const int cols = TN / S; // columns (rows of A) this CTA finishes: a power of two, at least 4
    const int q = warp & 3; // quarter of the tensor memory's lanes this warp may read
    const int row = q * 32 + lane;
    if (warp >= 2 && good) {
        // Partial sums travel as [source][4 columns][row] packs of four floats: a warp stores 512 contiguous bytes,
        // and the reader's lanes take consecutive rows.  An undivided K needs no exchange.
        const uint32_t base = smem_u32(smem) + (uint32_t)(split * cols * GS_BN + row * 4) * 4;
        const int shift = __ffs(cols) - 1;
        constexpr int CH = TN < 32 ? 16 : 32;
#pragma unroll 1
        for (int c0 = 0; c0 < TN; c0 += CH) {
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
                    const uint32_t owner = (uint32_t)(c0 + i) >> shift, c = (uint32_t)(c0 + i) & (cols - 1);
                    st_cluster_v4(map_to_cta(base + c * GS_BN * 4, owner), r[i], r[i + 1], r[i + 2], r[i + 3]);
                }
            }
        }
        tc_fence_before_sync();
    }
    if (S > 1)
        cluster_sync_all();
    else
        __syncthreads();
    if (S > 1 && warp >= 2 && live && !*abort_flag) {
        const uint32_t part = smem_u32(smem) + row * 16;
        if (S == 2)
            gs_reduce<2>(P, M, part, cols, tok0 + split * cols, n0, row);
        else if (S == 4)
            gs_reduce<4>(P, M, part, cols, tok0 + split * cols, n0, row);
        else
            gs_reduce<8>(P, M, part, cols, tok0 + split * cols, n0, row);
    }
    if (warp == 2) { // all reads of the accumulator lie in front of the last barrier
        tc_fence_after_sync();
        tmem_dealloc(tmem, L::TMEM_COLS);
    }
}

template <int TN>
void launch_small(const gemm_small_params& P, int tiles_n, int tiles_m, cudaStream_t st) {
    allow_smem<gemm_small_kernel<TN>>(gs_layout<TN>::TOTAL);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(tiles_n * P.splits, tiles_m);
    cfg.blockDim = dim3(GEMM_THREADS);
    cfg.dynamicSmemBytes = gs_layout<TN>::TOTAL;
    cfg.stream = st;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = P.splits;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    CUDA_CHECK(cudaLaunchKernelEx(&cfg, gemm_small_kernel<TN>, P));
}

struct small_plan {
    int tn, splits;
    double cycles; // estimate
};

// The split with the lowest estimate.  Measured on the pieces: a step of 64 takes a CTA's (16 + TN / 8) KB from the L2
// at 64 bytes per cycle and SM, whichever CTAs share the SM; start, exchange and output cost 4000 cycles and 32 per
// column (2048 x 1024 x 1 row 5 us, 128 rows 7 us, 256 rows 10 us), once for all CTAs that are resident together.
small_plan plan_small(int M, int N, int K, int sms) {
    const int kb = (K + GEMM_BK - 1) / GEMM_BK;
    small_plan best{ 16, 1, 1e30 };
    for (int tn = 16; tn <= 256; tn *= 2) {
        const int tiles = (N + GS_BN - 1) / GS_BN * ((M + tn - 1) / tn);
        const int resident = tn == 256 ? sms : 2 * sms;
        for (int s = 1; s <= std::min(8, tn / 4) && (s == 1 || kb / s >= 2); s *= 2) {
            const int ctas = tiles * s;
            if (tn == 256 && s > 1 && ctas > sms * 7 / 8) // clusters of one CTA per SM leave some SMs without one
                break;
            // CTAs that share an SM even out; one per SM runs in whole rounds
            const double load = tn == 256 ? (ctas + sms - 1) / sms : std::max(1.0, (double)ctas / sms);
            const double cycles = load * ((kb + s - 1) / s) * (256 + 2 * tn) + (ctas + resident - 1) / resident * (4000.0 + 32 * tn);
            if (cycles < 0.98 * best.cycles) // a finer cut has to gain something
                best = { tn, s, cycles };
        }
        if (tn >= M)
            break;
    }
    return best;
}

} // namespace

// Whether the kernel above is expected to be faster than CTA pairs on 256 x 256 tiles: up to 128 rows always, beyond that
// when the pairs would leave much of the chip idle.  In time the estimate above comes out as 1.25 times its cycles and 4600 for
// the launch; the pairs take 560 cycles per step of 64 and round of tiles and 14500 for launch, start and output.  The
// line this draws at 4096 x 4096 lies between 512 rows (23 us here, 30 us with pairs) and 768 (33 and 31), at 7168 x 2048
// between 200 rows (16.6 and 17.2) and 384 (20 and 18), at 4096 x 14336 between 512 (55 and 78) and 768 (80 and 78).
bool gemm_small_preferred(int M, int N, int K, int sms) {
    if (M <= 128)
        return true;
    const int tiles = ((M + 255) / 256) * ((N + 255) / 256), pairs = sms / 2, kb = (K + GEMM_BK - 1) / GEMM_BK;
    const int rounds = (tiles + pairs - 1) / pairs;
    return plan_small(M, N, K, sms).cycles * 1.25 + 4600 < (double)rounds * kb * 560 + 14500;
}

void gemm_bf16_small(const void* A, const void* B, void* C, int M, int N, int K, int epilogue, uint32_t* err, cudaStream_t st,
                     const int* rows_dev) {
    CCL_THROW_IF_NOT(M > 0 && N > 0 && K > 0 && N % 8 == 0 && K % 8 == 0, "unsupported GEMM shape ", M, "x", N, "x", K);
    const int sms = device_sms();
    const small_plan plan = plan_small(M, N, K, sms);
    gemm_small_params P;
    std::memset(&P, 0, sizeof(P));
    P.tmA = make_bf16_kmajor_map(A, M, K, plan.tn);
    P.tmB = make_bf16_kmajor_map(B, N, K, GS_BN);
    P.C = (__nv_bfloat16*)C;
    P.err = err;
    P.M = M;
    P.N = N;
    P.K = K;
    P.epilogue = epilogue;
    P.splits = plan.splits;
    P.rows = rows_dev;
    P.timeout_ns = (unsigned long long)env_data::get().wait_timeout_ms * 1000000ull;
    const int tiles_n = (N + GS_BN - 1) / GS_BN, tiles_m = (M + plan.tn - 1) / plan.tn;
    switch (plan.tn) {
        case 16: launch_small<16>(P, tiles_n, tiles_m, st); break;
        case 32: launch_small<32>(P, tiles_n, tiles_m, st); break;
        case 64: launch_small<64>(P, tiles_n, tiles_m, st); break;
        case 128: launch_small<128>(P, tiles_n, tiles_m, st); break;
        default: launch_small<256>(P, tiles_n, tiles_m, st); break;
    }
}

} // namespace gpu
} // namespace cclx
