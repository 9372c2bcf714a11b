// bf16 GEMM on CTA pairs: C[M,N] = A[M,K] * B[N,K]^T with tcgen05.mma.cta_group::2.
//
// Two CTAs of a cluster share one 256 x 256 output tile.  Each stages its own 128 rows of A and its
// own 128-row half of the B tile (32 KB per 64-deep K step instead of the 48 KB a single CTA needs
// for 128 x 256), which is what the L2 -> shared-memory path can sustain at full tensor rate.  The
// even CTA issues the MMAs for both; each CTA's tensor memory holds its 128 accumulator rows and its
// own epilogue warps drain them.  Tiles are visited in groups of columns, down the rows of a group: the group's part of B
// stays in the L2 while A streams past it once per group, so a group is as wide as a third of the L2 allows (8192 x
// 14336 x 4096: 14 columns instead of 8 take 2 % off the time under the power cap).
//
// Roles per CTA (576 threads): warp 0 TMA producer, warp 1 MMA issuer (leader CTA only), 16 epilogue warps (TMEM -> registers ->
// bf16 -> whole 32-byte sectors of the lanes' own rows).  With four of them and a transpose through shared memory, which the
// tensor cores and the copies keep busy, a tile's output took longer than 16 steps of K: 8192 x 4096 x 1024 with SiLU 59.1 us,
// now 53.4 (without 52.1 and 50.2; 1076 x 5648 x 560 13.8 and 13.0; 8192 x 14336 x 4096 739 and 726 under the power cap).
// Every mbarrier wait is bounded; the cluster barriers at start and end are reached on every path.
// The reference library has no GEMM: this kernel serves the tensor-parallel and expert-parallel layers.
#include <algorithm>
#include <atomic>
#include <cstring>

#include "core/env.hpp"
#include "core/log.hpp"
#include "gpu/cuda_driver.hpp"
#include "gpu/fused_gemm.cuh"
#include "gpu/fused_gemm.hpp"
#include "gpu/launch_util.cuh"
#include "gpu/row_store.cuh"

namespace cclx {
namespace gpu {

constexpr int G2_STAGES = 6;
constexpr int G2_BN = 256; // tile columns
constexpr int G2_HALF = 128; // rows of A and rows of B staged per CTA
constexpr int G2_STAGE_A = G2_HALF * GEMM_BK * 2;
constexpr int G2_STAGE_B = G2_HALF * GEMM_BK * 2;
constexpr int G2_RING = G2_STAGES * (G2_STAGE_A + G2_STAGE_B);
constexpr int G2_EPI_WARPS = 16;
constexpr int G2_PART = G2_BN / (G2_EPI_WARPS / 4); // columns of a tile that an epilogue warp drains
constexpr int G2_THREADS = 64 + 32 * G2_EPI_WARPS;
constexpr int G2_SMEM = 1024 + G2_RING + 256;
constexpr size_t G2_GROUP_BYTES = 32u << 20; // of B per raster group

struct gemm2_params {
    CUtensorMap tmA; // [M,K], box 64 x 128
    CUtensorMap tmB; // [N,K], box 64 x 128
    __nv_bfloat16* C;
    uint32_t* err;
    int M, N, K, epilogue;
    int group_n; // tile columns per raster group
    int trade; // lanes trade sectors before they store
    unsigned long long timeout_ns;
    const int* rows; // optional device word: only the first min(M, *rows) rows of A are multiplied
};

namespace {

__device__ __forceinline__ void g2_fail(const gemm2_params& P, volatile int* abort_flag, uint32_t code, uint32_t detail) {
    *abort_flag = 1;
    if (P.err && P.err[0] == GE_OK) {
        P.err[1] = blockIdx.x;
        P.err[2] = detail;
        __threadfence();
        P.err[0] = code;
    }
}

// tile index -> (row block of 256, column block of 256), groups of `group` columns
__device__ __forceinline__ void g2_tile(int t, int tiles_m, int tiles_n, int group, int& mi, int& ni) {
    const int per_group = group * tiles_m;
    const int grp = t / per_group, in = t % per_group;
    const int width = min(group, tiles_n - grp * group);
    mi = in / width;
    ni = grp * group + in % width;
}

// 2 W columns of rows row0 + lane of C from column `col` on, a multiple of 16, in whole 32-byte sectors.  Where N is an odd number of
// eights every other row begins in the middle of one: then each lane writes its own row, the first and the last half sector alone.
template <int W>
__device__ __forceinline__ void g2_store(const gemm2_params& P, int M, int row0, int col, int lane, uint32_t (&w)[W]) {
    if (P.trade) {
        store_rows(P.C, M, P.N, row0, col, lane, w);
        return;
    }
    const int row = row0 + lane;
    if (row >= M)
        return;
    __nv_bfloat16* p = P.C + (size_t)row * P.N + col;
    const int left = P.N - col; // columns, a multiple of 8
    if (((uintptr_t)p & 31) == 0) {
#pragma unroll
        for (int i = 0; i < W; i += 8) {
            if (2 * i + 16 <= left)
                st_16(p + 2 * i, w + i);
            else if (2 * i < left)
                st_8(p + 2 * i, w + i);
        }
    }
    else {
        if (left > 0)
            st_8(p, w);
#pragma unroll
        for (int i = 4; i + 8 < W; i += 8) {
            if (2 * i + 16 <= left)
                st_16(p + 2 * i, w + i);
            else if (2 * i < left)
                st_8(p + 2 * i, w + i);
        }
        if (2 * (W - 4) < left)
            st_8(p + 2 * (W - 4), w + W - 4);
    }
}

// PAIRS: CTA pairs per cluster.  With two, the tiles of a last, less than half full round are cut along K between the pairs of a
// cluster, which add their halves through distributed shared memory.
template <int PAIRS>
__global__ void __launch_bounds__(G2_THREADS, 1) gemm2sm_kernel(const __grid_constant__ gemm2_params P) {
    using namespace sm100;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = smem;
    uint8_t* sB = smem + G2_STAGES * G2_STAGE_A;
    uint64_t* bars = (uint64_t*)(smem + G2_RING);
    uint64_t* full = bars; // [STAGES]  used in the leader: bytes of both CTAs
    uint64_t* empty = bars + G2_STAGES; // [STAGES]  per CTA, signalled by the MMA commit
    uint64_t* tfull = bars + 2 * G2_STAGES; // [2] per CTA
    uint64_t* tempty = bars + 2 * G2_STAGES + 2; // [2] used in the leader: the epilogue warps of both CTAs
    uint32_t* tmem_holder = (uint32_t*)(bars + 2 * G2_STAGES + 4);
    volatile int* abort_flag = (volatile int*)(tmem_holder + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank(), pair = rank >> 1, cr = rank & 1; // cr 0: leader of its pair
    const bool leader = cr == 0;
    const int n_clusters = gridDim.x / (2 * PAIRS), cluster = blockIdx.x / (2 * PAIRS);
    const int n_pairs = n_clusters * PAIRS, me = cluster * PAIRS + (int)pair;
    const int KB = (P.K + GEMM_BK - 1) / GEMM_BK;
    const unsigned long long limit = P.timeout_ns;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < G2_STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], 2 * G2_EPI_WARPS);
        }
        mbar_fence_init();
        tma_prefetch_desc(&P.tmA);
        tma_prefetch_desc(&P.tmB);
    }
    if (warp == 2) {
        tmem_alloc_2sm(tmem_holder, 512);
        tc_fence_before_sync();
    }
    __syncthreads();
    cluster_sync_all(); // the peers' barriers exist before anything is signalled across the pair
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_holder;
    pdl_trigger(); // the next kernel's blocks may take the SMs that this one's leave
    pdl_wait(); // everything above overlaps the end of the kernel in front
    // the row count may live on the device (rows that a kernel in front of this one delivered): every thread
    // reads the same word, so all roles walk the same tiles
    const int M = P.rows ? max(0, min(P.M, *P.rows)) : P.M;
    const int tiles_m = (M + 255) / 256, tiles_n = (P.N + G2_BN - 1) / G2_BN;
    const int total_tiles = tiles_m * tiles_n;
    // tiles [whole, total_tiles) are cut in two, one per cluster
    static_assert(PAIRS == 1 || PAIRS == 2, "a tile is cut in two at most");
    const int left = PAIRS > 1 && KB > 1 ? total_tiles % n_pairs : 0;
    const int whole = left <= n_clusters ? total_tiles - left : total_tiles;
    const bool cut = whole + cluster < total_tiles; // the same in all CTAs of the cluster
    const int mine = me < whole ? (whole - me + n_pairs - 1) / n_pairs : 0; // uncut tiles of this pair
    auto tile_of = [&](int n) { return n < mine ? me + n * n_pairs : whole + cluster; };
    auto k_first = [&](int n) { return n < mine ? 0 : KB * (int)pair / PAIRS; };
    auto k_last = [&](int n) { return n < mine ? KB : KB * ((int)pair + 1) / PAIRS; };
    const int items = mine + (cut ? 1 : 0);

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            for (int n = 0; n < items && !*abort_flag; n++) {
                int mi, ni;
                g2_tile(tile_of(n), tiles_m, tiles_n, P.group_n, mi, ni);
                const int k1 = k_last(n);
                for (int kb = k_first(n); kb < k1; kb++, it++) {
                    const uint32_t st = it % G2_STAGES, ph = (it / G2_STAGES) & 1;
                    if (!mbar_wait(&empty[st], ph ^ 1, abort_flag, limit)) {
                        g2_fail(P, abort_flag, GE_MBAR_TIMEOUT, 2);
                        break;
                    }
                    if (leader)
                        mbar_expect_tx(&full[st], 2 * (G2_STAGE_A + G2_STAGE_B));
                    tma_load_2d_2sm(sA + st * G2_STAGE_A, &P.tmA, kb * GEMM_BK, mi * 256 + (int)cr * G2_HALF, &full[st]);
                    tma_load_2d_2sm(sB + st * G2_STAGE_B, &P.tmB, kb * GEMM_BK, ni * G2_BN + (int)cr * G2_HALF,
                                    &full[st]);
                }
            }
            if (leader) { // copies of both CTAs still in flight must land before the pair may exit
                const uint32_t first = it > (uint32_t)G2_STAGES ? it - G2_STAGES : 0;
                for (uint32_t i = first; i < it; i++)
                    mbar_wait(&full[i % G2_STAGES], (i / G2_STAGES) & 1, abort_flag, limit);
            }
        }
        __syncwarp();
    }
    else if (warp == 1) {
        if (lane == 0 && leader) {
            constexpr uint32_t idesc = make_idesc_bf16(256, G2_BN);
            const uint16_t both = (uint16_t)(3u << (2 * pair));
            uint32_t it = 0;
            for (int n = 0; n < items && !*abort_flag; n++) {
                const uint32_t acc = n & 1, aph = (n >> 1) & 1;
                if (!mbar_wait(&tempty[acc], aph ^ 1, abort_flag, limit)) {
                    g2_fail(P, abort_flag, GE_MBAR_TIMEOUT, 3);
                    break;
                }
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + acc * G2_BN;
                bool bad = false;
                const int k0 = k_first(n), k1 = k_last(n);
                for (int kb = k0; kb < k1; kb++, it++) {
                    const uint32_t st = it % G2_STAGES, ph = (it / G2_STAGES) & 1;
                    if (!mbar_wait(&full[st], ph, abort_flag, limit)) {
                        g2_fail(P, abort_flag, GE_MBAR_TIMEOUT, 4);
                        bad = true;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t a_addr = smem_u32(sA + st * G2_STAGE_A);
                    const uint32_t b_addr = smem_u32(sB + st * G2_STAGE_B);
#pragma unroll
                    for (int k = 0; k < GEMM_BK / GEMM_UMMA_K; k++)
                        umma_bf16_2sm(d_tmem, make_smem_desc_sw128(a_addr + k * GEMM_UMMA_K * 2),
                                      make_smem_desc_sw128(b_addr + k * GEMM_UMMA_K * 2), idesc, (kb != k0 || k != 0) ? 1u : 0u);
                    umma_commit_2sm(&empty[st], both); // both CTAs may refill the stage once these MMAs have read it
                }
                if (bad)
                    break;
                umma_commit_2sm(&tfull[acc], both); // accumulator complete in both CTAs
            }
        }
        __syncwarp();
    }
    const int q = warp & 3; // TMEM lane quarter this warp may read
    const int part = (warp - 2) >> 2; // this warp's share of the columns
    auto convert = [&](const uint32_t (&r)[16], uint32_t* w) { // activation and bf16
#pragma unroll
        for (int i = 0; i < 8; i++) {
            float a0 = __uint_as_float(r[2 * i]), a1 = __uint_as_float(r[2 * i + 1]);
            if (P.epilogue == EPI_SILU) {
                a0 = silu_f(a0);
                a1 = silu_f(a1);
            }
            const __nv_bfloat162 h = __floats2bfloat162_rn(a0, a1);
            w[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
    };
    bool good = warp >= 2;
    if (warp >= 2) {
        const uint32_t tempty_leader = smem_u32(&tempty[0]) & PEER_BIT_MASK;
        for (int n = 0; n < items && !warp_sees(abort_flag); n++) {
            const uint32_t acc = n & 1, aph = (n >> 1) & 1;
            good = mbar_wait_warp(&tfull[acc], aph, abort_flag, limit);
            if (!good) {
                if (lane == 0)
                    g2_fail(P, abort_flag, GE_MBAR_TIMEOUT, 5);
                break;
            }
            tc_fence_after_sync();
            if (n == mine) // the cut tile
                break;
            int mi, ni;
            g2_tile(tile_of(n), tiles_m, tiles_n, P.group_n, mi, ni);
            const int row0 = mi * 256 + (int)cr * G2_HALF + q * 32, col0 = ni * G2_BN + part * G2_PART;
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * G2_BN + part * G2_PART;
            uint32_t w[G2_PART / 2];
#pragma unroll
            for (int c = 0; c < G2_PART; c += 16) {
                uint32_t r[16];
                tmem_ld_32x16(taddr + c, r);
                tmem_ld_wait();
                if (c == G2_PART - 16) {
                    // all reads of this accumulator are done: hand it back to the leader's MMA warp
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive_cluster(tempty_leader + acc * 8);
                }
                convert(r, w + c / 2);
            }
            g2_store(P, M, row0, col0, lane, w);
            __syncwarp(); // lanes part where rows or columns end
        }
        __syncwarp();
    }
    if constexpr (PAIRS > 1) {
        if (cut) {
            // Pair p finishes columns [128 p, 128 p + 128) of the tile: the other pair's half sums of them arrive in the ring, which
            // nobody uses any more, as packs of four columns per row.  The sum of two halves does not depend on their order.
            constexpr int HALF_PART = G2_PART / 2;
            static_assert(G2_BN / 2 / 4 * G2_HALF * 16 <= G2_RING, "the half sums must fit the ring");
            const uint32_t acc = mine & 1;
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * G2_BN + part * HALF_PART;
            const uint32_t here = smem_u32(smem) + (uint32_t)(q * 32 + lane + part * (HALF_PART / 4) * G2_HALF) * 16;
            cluster_sync_all();
            if (warp >= 2 && good) {
                const uint32_t there = map_to_cta(here, rank ^ 2);
#pragma unroll
                for (int c = 0; c < HALF_PART; c += 16) {
                    uint32_t r[16];
                    tmem_ld_32x16(taddr + (pair ^ 1) * (G2_BN / 2) + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; i += 4)
                        st_cluster_v4(there + (uint32_t)(c + i) / 4 * G2_HALF * 16, r[i], r[i + 1], r[i + 2], r[i + 3]);
                }
            }
            cluster_sync_all();
            if (warp >= 2 && good && !warp_sees(abort_flag)) {
                int mi, ni;
                g2_tile(whole + cluster, tiles_m, tiles_n, P.group_n, mi, ni);
                uint32_t w[HALF_PART / 2];
#pragma unroll
                for (int c = 0; c < HALF_PART; c += 16) {
                    uint32_t r[16];
                    tmem_ld_32x16(taddr + pair * (G2_BN / 2) + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; i += 4) {
                        float v[4];
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                                     : "r"(here + (uint32_t)(c + i) / 4 * G2_HALF * 16));
#pragma unroll
                        for (int k = 0; k < 4; k++)
                            r[i + k] = __float_as_uint(__uint_as_float(r[i + k]) + v[k]);
                    }
                    convert(r, w + c / 2);
                }
                g2_store(P, M, mi * 256 + (int)cr * G2_HALF + q * 32, ni * G2_BN + (int)pair * (G2_BN / 2) + part * HALF_PART, lane, w);
            }
        }
    }

    // converge: nobody leaves while the partner may still read its shared memory or signal its barriers
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync_all();
    if (warp == 2) {
        tc_fence_after_sync();
        tmem_dealloc_2sm(tmem_base, 512);
    }
}

// clusters of `PAIRS` CTA pairs that fit the device
template <int PAIRS>
int most_clusters() {
    allow_smem<gemm2sm_kernel<PAIRS>>(G2_SMEM);
    static std::atomic<int> known[64];
    int dev = 0;
    CUDA_CHECK(cudaGetDevice(&dev));
    int n = dev < 64 ? known[dev].load(std::memory_order_relaxed) : 0;
    if (n == 0) {
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr{};
        cfg.gridDim = dim3(2 * PAIRS);
        cfg.blockDim = dim3(G2_THREADS);
        cfg.dynamicSmemBytes = G2_SMEM;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2 * PAIRS;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        CUDA_CHECK(cudaOccupancyMaxActiveClusters(&n, gemm2sm_kernel<PAIRS>, &cfg));
        n = std::max(n, 1);
        if (dev < 64)
            known[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

// Expected time in us: 5.6 for launch, start and output, 0.35 per step of 64 and round of tiles, a sixth more where the rows of a
// box begin between the 32-byte sectors; clusters of two pairs start 1.2 later, a cut tile takes half a round and 1.0 for the
// exchange (rms of 13 % over 150 products).  4096 x 4096 with 512 rows, 32 tiles: 26.3 us uncut, 19.1 cut; with 1024 rows, 64 tiles
// for 74 pairs, nothing is cut.  Clusters of four leave some SMs out, so products of many rounds keep the pairs.
double estimate(int M, int N, int K, int pairs) {
    const double step = (K % 16 ? 1.165 : 1.0) * 0.35 * ((K + GEMM_BK - 1) / GEMM_BK);
    const long long tiles = (long long)((M + 255) / 256) * ((N + G2_BN - 1) / G2_BN);
    if (pairs == 1) {
        const int most = device_sms() / 2;
        return 5.6 + (tiles + most - 1) / most * step;
    }
    const long long clusters = std::min<long long>(most_clusters<2>(), tiles), left = tiles % (2 * clusters);
    const bool cut = left > 0 && left <= clusters;
    return 6.8 + (tiles / (2 * clusters) + (cut ? 0.5 : left > 0 ? 1.0 : 0.0)) * step + (cut ? 1.0 : 0);
}

template <int PAIRS>
void launch_2sm(const gemm2_params& P, int clusters, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * PAIRS * clusters);
    cfg.blockDim = dim3(G2_THREADS);
    cfg.dynamicSmemBytes = G2_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2 * PAIRS;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    CUDA_CHECK(cudaLaunchKernelEx(&cfg, gemm2sm_kernel<PAIRS>, P));
}

} // namespace

void gemm_bf16_2sm(const void* A, const void* B, void* C, int M, int N, int K, int epilogue, int clusters,
                   uint32_t* err, cudaStream_t st, const int* rows_dev, int pairs) {
    CCL_THROW_IF_NOT(M > 0 && N > 0 && K > 0 && N % 8 == 0 && K % 8 == 0, "unsupported GEMM shape ", M, "x", N, "x", K);
    CCL_THROW_IF_NOT(((uintptr_t)C & 15) == 0, "GEMM output must be 16-byte aligned");
    allow_smem<gemm2sm_kernel<1>>(G2_SMEM);
    allow_smem<gemm2sm_kernel<2>>(G2_SMEM);
    gemm2_params P;
    std::memset(&P, 0, sizeof(P));
    P.tmA = make_bf16_map(A, M, K, G2_HALF);
    P.tmB = make_bf16_map(B, N, K, G2_HALF);
    P.C = (__nv_bfloat16*)C;
    P.err = err;
    P.M = M;
    P.N = N;
    P.K = K;
    P.epilogue = epilogue;
    P.rows = rows_dev;
    // Rows that begin at a sector, but not at a 128-byte line: a lane's 64 columns lie in two lines then.  5728 x 5616 x 6024 387 us,
    // 379 with the trade, 2966 x 12240 x 904 77.8 and 76.1.  Rows of whole lines are better off without: 8192 x 4096 x 4096 201 and
    // 204 with it, under the power cap.
    P.trade = N % 16 == 0 && N % 64 != 0 && ((uintptr_t)C & 31) == 0;
    P.timeout_ns = (unsigned long long)env_data::get().wait_timeout_ms * 1000000ull;
    const int tiles_n = (N + G2_BN - 1) / G2_BN;
    const int most = (int)std::min<size_t>(std::max<size_t>(G2_GROUP_BYTES / ((size_t)G2_BN * K * 2), 4), 32);
    const int groups = (tiles_n + most - 1) / most;
    P.group_n = (tiles_n + groups - 1) / groups; // groups of about the same width
    const int tiles = ((M + 255) / 256) * tiles_n;
    if (clusters == 0 && pairs == 2)
        launch_2sm<2>(P, std::min(most_clusters<2>(), tiles), st);
    else
        launch_2sm<1>(P, std::max(1, std::min(clusters > 0 ? clusters : device_sms() / 2, tiles)), st);
}

double gemm_2sm_estimate(int M, int N, int K, int pairs) {
    return estimate(M, N, K, pairs);
}

} // namespace gpu
} // namespace cclx
