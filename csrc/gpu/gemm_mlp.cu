// The products on both sides of a GELU on CTA pairs (tcgen05.mma.cta_group::2, 256 x 256 tiles, see gemm_2sm.cu), with the
// activation in their epilogues:
//
//   forward : u = x W1^T + b1 and gelu(u), both written from one accumulator;
//   backward: du = (dy W2) gelu'(u) and the sums of du over the rows, the gradient of b1.
//
// As a pass of its own the GELU reads and writes 128 MB for 8192 x 4096 values, its gradient 192 MB; here the backward
// product reads u where it would have waited for tensor cores, and nothing else moves.  W2 lies as [K, N]: its tiles are
// staged with N along the 128-byte rows (64 columns each) and multiplied as an MN-major operand, so nothing is transposed.
//
// Sixteen epilogue warps per CTA, four on each quarter of the tensor memory's lanes, since latency is what an activation costs
// (with eight, 0.35 instructions per scheduler and cycle).  They read and write whole 32-byte sectors of their lanes' rows and
// work on pairs of values.  8192 x 4096 x 1024: forward 59 us where product and pass took 51 and 19.5, backward 67 us where they
// took 50 and 34; both with the products around them 326 us instead of 369.  The plain product takes 50: two outputs, or u beside
// the product, are what is left.
#include <algorithm>
#include <cstring>

#include "capi/capi_common.hpp"
#include "core/env.hpp"
#include "core/log.hpp"
#include "gpu/cuda_driver.hpp"
#include "gpu/f32x2.cuh"
#include "gpu/fused_gemm.cuh"
#include "gpu/gelu.cuh"
#include "gpu/launch_util.cuh"
#include "gpu/row_store.cuh"

namespace cclx {
namespace gpu {

namespace {

constexpr int GM_STAGES = 6;
constexpr int GM_BN = 256; // tile columns
constexpr int GM_HALF = 128; // rows of A and columns of B staged per CTA
constexpr int GM_STAGE = GM_HALF * GEMM_BK * 2; // of one operand
constexpr int GM_RING = GM_STAGES * 2 * GM_STAGE;
constexpr int GM_EPI_WARPS = 16;
constexpr int GM_THREADS = 64 + 32 * GM_EPI_WARPS;
constexpr int GM_SUMS = 2 * 4 * GM_BN * 4; // column sums of two tiles, by quarter
constexpr int GM_SMEM = 1024 + GM_RING + GM_SUMS + 256;
constexpr size_t GM_GROUP_BYTES = 32u << 20; // of B per raster group

struct mlp_params {
    CUtensorMap tmA; // [M,K], box 64 x 128
    CUtensorMap tmB; // forward [N,K], box 64 x 128; backward [K,N], box 64 x 64
    const __nv_bfloat16* bias; // forward: [N]
    __nv_bfloat16* u; // [M,N]: written by the forward product, read by the backward one
    __nv_bfloat16* out; // [M,N]: gelu(u), or du
    float* partial; // backward: [ceil(M / 128)][N] sums over 128 rows
    int M, N, K, group_n;
    int wide; // rows of u and out begin at 32-byte sectors
    unsigned long long timeout_ns;
};

// shared-memory descriptor of a bf16 operand staged as blocks of 64 columns: row k of a block is 128 bytes (128-byte swizzle), 8
// rows are 1024 bytes (stride byte offset), blocks are 64 rows = 8192 bytes apart (leading byte offset)
__device__ __forceinline__ uint64_t desc_mn_major(uint32_t smem_addr) {
    uint64_t d = (smem_addr & 0x3FFFF) >> 4;
    d |= (uint64_t)(8192 >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46; // descriptor version for sm_100
    d |= (uint64_t)2 << 61; // SWIZZLE_128B
    return d;
}

// sums 16 values per lane over the warp: lanes 2 l and 2 l + 1 end with the total of value l (16 exchanges)
__device__ __forceinline__ float warp_totals(float (&v)[16], int lane) {
#pragma unroll
    for (int n = 8; n > 0; n >>= 1) {
        const bool up = lane & 2 * n;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * n);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ f32x2 pair_of(uint32_t w) { // bf16 is the upper half of an fp32 word
    return pair(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

template <bool BWD>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GM_THREADS, 1) mlp_kernel(const __grid_constant__ mlp_params P) {
    using namespace sm100;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = smem;
    uint8_t* sB = smem + GM_STAGES * GM_STAGE;
    float* sums = (float*)(smem + GM_RING); // [tile parity][quarter][column]
    uint64_t* bars = (uint64_t*)(smem + GM_RING + GM_SUMS);
    uint64_t* full = bars; // [STAGES]  used in the leader: bytes of both CTAs
    uint64_t* empty = bars + GM_STAGES; // [STAGES]  per CTA, signalled by the MMA commit
    uint64_t* tfull = bars + 2 * GM_STAGES; // [2] per CTA
    uint64_t* tempty = bars + 2 * GM_STAGES + 2; // [2] used in the leader: the epilogue warps of both CTAs
    uint32_t* tmem_holder = (uint32_t*)(bars + 2 * GM_STAGES + 4);
    volatile int* abort_flag = (volatile int*)(tmem_holder + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t cr = cluster_ctarank(); // 0 = leader
    const bool leader = cr == 0;
    const int n_clusters = gridDim.x >> 1, cluster = blockIdx.x >> 1;
    const int KB = (P.K + GEMM_BK - 1) / GEMM_BK;
    const unsigned long long limit = P.timeout_ns;

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < GM_STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], 2 * GM_EPI_WARPS);
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
    cluster_sync_all(); // the peer's barriers exist before anything is signalled across the pair
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_holder;
    pdl_wait(); // everything above overlaps the end of the kernel in front
    const int tiles_m = (P.M + 255) / 256, tiles_n = (P.N + GM_BN - 1) / GM_BN;
    const int total_tiles = tiles_m * tiles_n;
    // groups of `group_n` tile columns, down the rows of a group (gemm_2sm.cu)
    auto tile_at = [&](int t, int& mi, int& ni) {
        const int per_group = P.group_n * tiles_m, grp = t / per_group, in = t % per_group;
        const int width = min(P.group_n, tiles_n - grp * P.group_n);
        mi = in / width;
        ni = grp * P.group_n + in % width;
    };

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            for (int t = cluster; t < total_tiles && !*abort_flag; t += n_clusters) {
                int mi, ni;
                tile_at(t, mi, ni);
                for (int kb = 0; kb < KB; kb++, it++) {
                    const uint32_t st = it % GM_STAGES, ph = (it / GM_STAGES) & 1;
                    if (!mbar_wait(&empty[st], ph ^ 1, abort_flag, limit)) {
                        *abort_flag = 1;
                        break;
                    }
                    if (leader)
                        mbar_expect_tx(&full[st], 4 * GM_STAGE);
                    uint8_t *a = sA + st * GM_STAGE, *b = sB + st * GM_STAGE;
                    const int n0 = ni * GM_BN + (int)cr * GM_HALF;
                    tma_load_2d_2sm(a, &P.tmA, kb * GEMM_BK, mi * 256 + (int)cr * GM_HALF, &full[st]);
                    if (BWD) {
                        tma_load_2d_2sm(b, &P.tmB, n0, kb * GEMM_BK, &full[st]);
                        tma_load_2d_2sm(b + GM_STAGE / 2, &P.tmB, n0 + 64, kb * GEMM_BK, &full[st]);
                    }
                    else
                        tma_load_2d_2sm(b, &P.tmB, kb * GEMM_BK, n0, &full[st]);
                }
            }
            if (leader) { // copies of both CTAs still in flight must land before the pair may exit
                const uint32_t first = it > (uint32_t)GM_STAGES ? it - GM_STAGES : 0;
                for (uint32_t i = first; i < it; i++)
                    mbar_wait(&full[i % GM_STAGES], (i / GM_STAGES) & 1, abort_flag, limit);
            }
        }
        __syncwarp();
    }
    else if (warp == 1) {
        if (lane == 0 && leader) {
            constexpr uint32_t idesc = make_idesc_bf16(256, GM_BN) | (BWD ? 1u << 16 : 0u); // bit 16: B is MN-major
            uint32_t it = 0, tc = 0;
            for (int t = cluster; t < total_tiles && !*abort_flag; t += n_clusters, tc++) {
                const uint32_t acc = tc & 1, aph = (tc >> 1) & 1;
                if (!mbar_wait(&tempty[acc], aph ^ 1, abort_flag, limit)) {
                    *abort_flag = 1;
                    break;
                }
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + acc * GM_BN;
                bool bad = false;
                for (int kb = 0; kb < KB; kb++, it++) {
                    const uint32_t st = it % GM_STAGES, ph = (it / GM_STAGES) & 1;
                    if (!mbar_wait(&full[st], ph, abort_flag, limit)) {
                        *abort_flag = 1;
                        bad = true;
                        break;
                    }
                    tc_fence_after_sync();
                    const uint32_t a_addr = smem_u32(sA + st * GM_STAGE), b_addr = smem_u32(sB + st * GM_STAGE);
#pragma unroll
                    for (int k = 0; k < GEMM_BK / GEMM_UMMA_K; k++)
                        umma_bf16_2sm(d_tmem, make_smem_desc_sw128(a_addr + k * GEMM_UMMA_K * 2),
                                      BWD ? desc_mn_major(b_addr + k * GEMM_UMMA_K * 128)
                                          : make_smem_desc_sw128(b_addr + k * GEMM_UMMA_K * 2),
                                      idesc, (kb | k) != 0 ? 1u : 0u);
                    umma_commit_2sm(&empty[st], 3); // both CTAs may refill the stage once these MMAs have read it
                }
                if (bad)
                    break;
                umma_commit_2sm(&tfull[acc], 3); // accumulator complete in both CTAs
            }
        }
        __syncwarp();
    }
    else {
        const int q = warp & 3; // TMEM lane quarter this warp may read
        const int c0 = (warp - 2) >> 2; // this warp's quarter of the columns
        const uint32_t tempty_leader = smem_u32(&tempty[0]) & PEER_BIT_MASK;
        bool ok = true; // a wait that ran out makes the outputs NaN: nobody reads an error word in the middle of a step
        // 16 columns of a lane's own row, a whole 32-byte sector: no pass through shared memory, which the tensor cores and
        // the copies keep busy
        auto load = [&](const __nv_bfloat16* m, int row, int col, uint32_t* w) {
            const __nv_bfloat16* p = m + (size_t)row * P.N + col;
            const bool on = row < P.M && col < P.N;
            if (P.wide && on)
                asm volatile("ld.global.L1::no_allocate.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                             : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
                             : "l"(p)
                             : "memory");
            else
#pragma unroll
                for (int h = 0; h < 8; h += 4) {
                    const uint4 x = on && col + h * 2 < P.N ? *reinterpret_cast<const uint4*>(p + h * 2) : make_uint4(0, 0, 0, 0);
                    w[h] = x.x;
                    w[h + 1] = x.y;
                    w[h + 2] = x.z;
                    w[h + 3] = x.w;
                }
        };
        auto store = [&](__nv_bfloat16* m, int row, int col, const uint32_t (&v)[8]) {
            __nv_bfloat16* p = m + (size_t)row * P.N + col;
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
                w[i] = ok ? v[i] : 0x7fc07fc0u;
            const bool on = row < P.M && col < P.N;
            if (P.wide) {
                if (on)
                    st_16(p, w);
            }
            else
#pragma unroll
                for (int h = 0; h < 8; h += 4)
                    if (on && col + h * 2 < P.N)
                        st_8(p + h * 2, w + h);
        };
        uint32_t tc = 0;
        // all of these warps see every tile, whatever happens to the other roles: they meet at a barrier
        for (int t = cluster; t < total_tiles; t += n_clusters, tc++) {
            int mi, ni;
            tile_at(t, mi, ni);
            const uint32_t acc = tc & 1, aph = (tc >> 1) & 1;
            const int row = mi * 256 + (int)cr * GM_HALF + q * 32 + lane, col0 = ni * GM_BN + c0 * 64;
            uint32_t in[32]; // this lane's part of u, or of the bias: on its way while the tensor cores work
#pragma unroll
            for (int c = 0; c < 64; c += 16) {
                if (BWD)
                    load(P.u, row, col0 + c, in + c / 2);
                else
#pragma unroll
                    for (int i = 0; i < 8; i += 4) {
                        const int n = col0 + c + i * 2;
                        const uint4 b = n < P.N ? __ldg(reinterpret_cast<const uint4*>(P.bias + n)) : make_uint4(0, 0, 0, 0);
                        in[c / 2 + i] = b.x;
                        in[c / 2 + i + 1] = b.y;
                        in[c / 2 + i + 2] = b.z;
                        in[c / 2 + i + 3] = b.w;
                    }
            }
            if (!mbar_wait_warp(&tfull[acc], aph, abort_flag, limit)) {
                *abort_flag = 1;
                ok = false;
            }
            tc_fence_after_sync();
#pragma unroll
            for (int c = 0; c < 64; c += 16) {
                const uint32_t* x = in + c / 2;
                uint32_t r[16], o[8];
                __syncwarp(); // lanes part where rows or columns end
                tmem_ld_32x16(tmem_base + ((uint32_t)(q * 32) << 16) + acc * GM_BN + c0 * 64 + c, r);
                tmem_ld_wait();
                if (c == 48) {
                    // all reads of this accumulator are done: hand it back to the leader's MMA warp
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive_cluster(tempty_leader + acc * 8);
                }
                if constexpr (BWD) {
                    float v[16];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        // the gradient of gelu(u) in bf16, as a product of its own would have left it
                        const uint32_t g = pack2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
                        unpair(mul2(pair_of(g), gelu_slope(pair_of(x[i]))), v[2 * i], v[2 * i + 1]);
                        o[i] = pack2(v[2 * i], v[2 * i + 1]);
                    }
                    store(P.out, row, col0 + c, o);
                    const float total = warp_totals(v, lane);
                    if ((lane & 1) == 0)
                        sums[((tc & 1) * 4 + q) * GM_BN + c0 * 64 + c + lane / 2] = ok ? total : __uint_as_float(0x7fc00000u);
                }
                else {
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        float lo, hi;
                        unpair(add2(pair(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1])), pair_of(x[i])), lo, hi);
                        o[i] = pack2(lo, hi);
                    }
                    store(P.u, row, col0 + c, o);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const f32x2 a = pair_of(o[i]);
                        float lo, hi;
                        unpair(mul2(a, gelu_gate(a)), lo, hi);
                        o[i] = pack2(lo, hi);
                    }
                    store(P.out, row, col0 + c, o);
                }
            }
            if (BWD) {
                // the quarters' sums meet once per tile, in a fixed order; the other parity's are free again by then
                dev::named_bar_sync(1, 32 * GM_EPI_WARPS);
                const int i = (warp - 2) * 32 + lane, n = ni * GM_BN + i;
                const float* s = sums + (tc & 1) * 4 * GM_BN + i;
                const int r = mi * 2 + (int)cr;
                if (i < GM_BN && n < P.N && r * GM_HALF < P.M)
                    P.partial[(size_t)r * P.N + n] = (s[0] + s[GM_BN]) + (s[2 * GM_BN] + s[3 * GM_BN]);
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

template <bool BWD>
void launch_mlp(const void* a, const void* b, const void* bias, void* u, void* out, float* partial, int M, int N, int K,
                cudaStream_t st) {
    CCL_THROW_IF_NOT(M > 0 && N > 0 && K > 0 && N % 8 == 0 && K % 8 == 0, "unsupported GEMM shape ", M, "x", N, "x", K);
    allow_smem<mlp_kernel<BWD>>(GM_SMEM);
    mlp_params P;
    std::memset(&P, 0, sizeof(P));
    P.tmA = make_bf16_map(a, M, K, GM_HALF);
    P.tmB = BWD ? make_bf16_map(b, K, N, 64) : make_bf16_map(b, N, K, GM_HALF);
    P.bias = (const __nv_bfloat16*)bias;
    P.u = (__nv_bfloat16*)u;
    P.out = (__nv_bfloat16*)out;
    P.partial = partial;
    P.M = M;
    P.N = N;
    P.K = K;
    P.wide = N % 16 == 0 && (((uintptr_t)u | (uintptr_t)out) & 31) == 0;
    P.timeout_ns = (unsigned long long)env_data::get().wait_timeout_ms * 1000000ull;
    const int tiles_n = (N + GM_BN - 1) / GM_BN, tiles = (M + 255) / 256 * tiles_n;
    const int most = (int)std::min<size_t>(std::max<size_t>(GM_GROUP_BYTES / ((size_t)GM_BN * K * 2), 4), 32);
    const int groups = (tiles_n + most - 1) / most;
    P.group_n = (tiles_n + groups - 1) / groups; // groups of about the same width
    launch_dependent(mlp_kernel<BWD>, dim3(2 * std::max(1, std::min(device_sms() / 2, tiles))), dim3(GM_THREADS), GM_SMEM, st, P);
}

} // namespace
} // namespace gpu
} // namespace cclx

using namespace cclx;

// *answer: 0 if the products with the activation inside may not run (no CTA pairs), 1 if they may, 2 if they are expected to be faster
// than library products and passes of their own: if the result fills at least three quarters of the rounds of tiles and its rows begin
// at 32-byte sectors.  Forward and backward of 8192 x 1024 x 4096 (rows, width, hidden width; 0.99 of seven rounds) 322 against
// 370 us, 2048 x 512 x 2048 (0.86 of one) 49.7 against 50.9, 666 x 1280 x 5120 (0.70 of one, though its tiles fill 0.81) 75.6 against
// 73.7, 300 x 4096 x 16384 (0.51 of two) 291 against 262; between sectors, 8192 x 768 x 3064 270 against 238, 2048 x 1024 x 4104 113
// against 108.  Of 119 sizes of 300 to 16384 rows and widths of 64 to 4096 the line gives up two that gained more than 2 % (4096 and
// 8192 x 1600 x 1600, 0.68, 5 and 7 %); of the 102 on this side three lose more than 1.5 % (666 x 3072 x 12288 2.5 %).
CCLX_API int cclx_mlp_preferred(int M, int N, int* answer) {
    return capi::guard([&] {
        *answer = 0;
        if (!env_data::get().gemm_2sm)
            return;
        const long long tiles = (M + 255ll) / 256 * ((N + 255) / 256), pairs = std::max(1, gpu::device_sms() / 2);
        const double room = 65536.0 * pairs * ((tiles + pairs - 1) / pairs);
        *answer = N % 16 == 0 && (double)M * N >= 0.75 * room ? 2 : 1;
    });
}

// u = x W1^T + bias and g = gelu(u): x [M,K], W1 [N,K], bias [N], u and g [M,N]; bf16, 16-byte aligned
CCLX_API int cclx_linear_gelu(const void* x, const void* w1, const void* bias, void* u, void* g, int M, int N, int K, void* stream) {
    return capi::guard([&] { gpu::launch_mlp<false>(x, w1, bias, u, g, nullptr, M, N, K, (cudaStream_t)stream); });
}

// rows of N floats that cclx_linear_gelu_bwd leaves in `partial`
CCLX_API int cclx_linear_gelu_bwd_rows(int M) {
    return (M + gpu::GM_HALF - 1) / gpu::GM_HALF;
}

// du = (dy W2) gelu'(u): dy [M,K], W2 [K,N], u and du [M,N]; `partial` receives the sums of du over 128 rows each, in fp32
CCLX_API int cclx_linear_gelu_bwd(const void* dy, const void* w2, const void* u, void* du, float* partial, int M, int N, int K,
                                  void* stream) {
    return capi::guard([&] { gpu::launch_mlp<true>(dy, w2, nullptr, (void*)u, du, partial, M, N, K, (cudaStream_t)stream); });
}
