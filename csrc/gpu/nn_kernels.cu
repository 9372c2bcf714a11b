// Memory-bound layer kernels of the transformer blocks used by the data-parallel training path:
// LayerNorm forward / backward (input gradient plus the weight and bias gradients in the same pass),
// column sums for bias gradients, and the strided copies that assemble a packed QKV gradient.
// The reference is a communication library and has no such kernels; they exist because the training
// step that the gradient allreduce overlaps with is otherwise dominated by framework kernels that
// re-read activations several times.  All math in fp32, bf16 storage.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "capi/capi_common.hpp"
#include "core/log.hpp"
#include "gpu/async_copy.cuh"
#include "gpu/cuda_driver.hpp"
#include "gpu/f32x2.cuh"
#include "gpu/gelu.cuh"
#include "gpu/launch_util.cuh"

using namespace cclx;
using namespace cclx::gpu;

namespace {

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ void unpack8(const uint4& u, float (&x)[8]) {
    const uint32_t w[4] = { u.x, u.y, u.z, u.w };
#pragma unroll
    for (int i = 0; i < 4; i++) { // bf16 is the upper half of an fp32 word
        x[2 * i] = __uint_as_float(w[i] << 16);
        x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// y = (x - mean) * rstd * w + b ; optionally x = x + residual first (the sum is written to `sum_out`).
//
// Bound by memory: x (and the residual) in, y (and the sum) out.  One warp owns a row, lane l holds the 16-byte packs
// l, l + 32, ... of it (V = packs per lane, the last one partial when the width is no multiple of 256), so the two
// reductions are shuffles and nothing synchronises.  The row stays packed while it waits and gamma / beta are
// re-read from L1 for every row, which leaves enough warps per SM to keep the loads of some 20 rows in flight.
template <int V>
__global__ void __launch_bounds__(128) ln_fwd_kernel(const uint4* __restrict__ x, const uint4* __restrict__ res,
                                                     const uint4* __restrict__ w, const uint4* __restrict__ b,
                                                     uint4* __restrict__ y, uint4* __restrict__ sum_out,
                                                     float* __restrict__ mean, float* __restrict__ rstd, size_t rows,
                                                     int packs, float inv_d, float eps) {
    const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const bool last_on = lane + (V - 1) * 32 < packs;
    for (size_t r = (size_t)blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += (size_t)gridDim.x * wpb) {
        const size_t base = r * packs + lane;
        uint4 u[V], q[V];
#pragma unroll
        for (int v = 0; v < V; v++)
            u[v] = v < V - 1 || last_on ? x[base + v * 32] : make_uint4(0, 0, 0, 0);
        float s = 0.f;
        if (res) {
#pragma unroll
            for (int v = 0; v < V; v++)
                q[v] = v < V - 1 || last_on ? res[base + v * 32] : make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int v = 0; v < V; v++) {
                float a[8], c[8];
                unpack8(u[v], a);
                unpack8(q[v], c);
#pragma unroll
                for (int e = 0; e < 8; e++)
                    a[e] += c[e];
                u[v] = pack8(a); // the sum lives in bf16
                if (v < V - 1 || last_on)
                    sum_out[base + v * 32] = u[v];
            }
        }
#pragma unroll
        for (int v = 0; v < V; v++) {
            float a[8];
            unpack8(u[v], a);
#pragma unroll
            for (int e = 0; e < 8; e++)
                s += a[e];
        }
        const float m = warp_sum_f(s) * inv_d;
        float var = 0.f;
#pragma unroll
        for (int v = 0; v < V; v++) {
            float a[8];
            unpack8(u[v], a);
            if (v < V - 1 || last_on) {
#pragma unroll
                for (int e = 0; e < 8; e++)
                    var = fmaf(a[e] - m, a[e] - m, var);
            }
        }
        const float rs = rsqrtf(warp_sum_f(var) * inv_d + eps);
#pragma unroll
        for (int v = 0; v < V; v++) {
            if (v < V - 1 || last_on) {
                float a[8], wv[8], bv[8];
                unpack8(u[v], a);
                unpack8(__ldg(w + lane + v * 32), wv);
                unpack8(__ldg(b + lane + v * 32), bv);
#pragma unroll
                for (int e = 0; e < 8; e++)
                    a[e] = fmaf((a[e] - m) * rs, wv[e], bv[e]);
                y[base + v * 32] = pack8(a);
            }
        }
        if (lane == 0) {
            mean[r] = m;
            rstd[r] = rs;
        }
    }
}

// Sums NV values over the warp at once: each exchange halves the number of values a lane still carries, so 8 values
// take 9 shuffles instead of 40.  Lane l ends with the total of value (l * NV / 32).
template <int NV>
__device__ __forceinline__ float warp_sum_many(float (&v)[NV], int lane) {
#pragma unroll
    for (int n = NV / 2, o = 16; n > 0; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n; i++) {
            const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int o = 16 / NV; o > 0; o >>= 1)
        v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

constexpr int LN_BWD_ROWS = 2; // rows per step of a group
constexpr int LN_BWD_STAGES = 4; // steps in flight or in use
constexpr int LN_BWD_BLOCKS = 2; // resident blocks per SM

// dx = rstd * (g - mean(g) - xhat * mean(g * xhat)), g = dy * w;  partial dgamma / dbeta (and column sums of dx) per
// block.  `dres` (optional) is added to dx: the gradient that reached the residual branch.
//
// Bound by memory: dy, x, dres in, dx out.  A thread owns 8 columns (one 16-byte pack) of every row its group of `tpr`
// threads works on, so the column sums cost 8 registers each, and a group takes R rows per step: one block barrier
// per R rows (the row sums cross the warps of a group through shared memory, double-buffered).  Every thread
// copies its own packs of the next three steps into shared memory with cp.async and reads back only those, so no
// barrier guards the ring and 147 KB per SM are in flight whatever the registers hold.  The instruction rate is the next limit (0.74 issued per
// scheduler and cycle with scalar arithmetic), hence the packed pairs.  A warp per row with the whole
// row and its column sums in registers needed 191 of them, had 8 warps per SM and ran at half the copy rate.
template <int R, bool COLSUM>
__global__ void __launch_bounds__(256, LN_BWD_BLOCKS)
    ln_bwd_kernel(const uint4* __restrict__ dy, const uint4* __restrict__ x, const uint4* __restrict__ w,
                  const float* __restrict__ mean, const float* __restrict__ rstd, const uint4* __restrict__ dres,
                  uint4* __restrict__ dx, float* __restrict__ partial, size_t rows, int packs, int tpr, float inv_d) {
    constexpr int NS = COLSUM ? 3 : 2;
    extern __shared__ __align__(16) float sh[]; // ring, then the row sums; the block's column sums at the end
    const int groups = blockDim.x / tpr;
    const int grp = threadIdx.x / tpr, c = threadIdx.x - grp * tpr;
    const int lane = threadIdx.x & 31, gw = c >> 5;
    const bool on = c < packs;
    uint4* ring = reinterpret_cast<uint4*>(sh); // [stage][tensor][row][thread]
    float* sums = sh + (size_t)LN_BWD_STAGES * 3 * R * blockDim.x * 4; // [2][group][2 R][8]: up to 8 warps' shares, zeros behind
    for (int i = threadIdx.x; i < 2 * groups * 2 * R * 8; i += blockDim.x)
        sums[i] = 0.f;
    __syncthreads();
    pdl_trigger(); // the final sum may be scheduled as soon as SMs fall idle; it waits for this grid's end
    f32x2 wv[4], acc2[NS][4];
    unpack4x2(on ? w[c] : make_uint4(0, 0, 0, 0), wv);
#pragma unroll
    for (int i = 0; i < NS; i++)
#pragma unroll
        for (int e = 0; e < 4; e++)
            acc2[i][e] = 0;
    const size_t step = (size_t)gridDim.x * groups * R;
    const size_t first = ((size_t)blockIdx.x * groups + grp) * R;
    auto at = [&](int stage, int tensor, int k) { return ring + ((size_t)(stage * 3 + tensor) * R + k) * blockDim.x + threadIdx.x; };
    auto fetch = [&](size_t r0, int stage) { // rows behind the end arrive as zeros
#pragma unroll
        for (int k = 0; k < R; k++) {
            const bool ok = on && r0 + k < rows;
            const size_t i = ok ? (r0 + k) * packs + c : 0;
            copy16_async(at(stage, 0, k), x + i, ok);
            copy16_async(at(stage, 1, k), dy + i, ok);
            if (dres)
                copy16_async(at(stage, 2, k), dres + i, ok);
        }
        copy_commit();
    };
    float m[R], rs[R];
    auto fetch_stats = [&](size_t r0) {
#pragma unroll
        for (int k = 0; k < R; k++) {
            m[k] = r0 + k < rows ? mean[r0 + k] : 0.f;
            rs[k] = r0 + k < rows ? rstd[r0 + k] : 0.f;
        }
    };
#pragma unroll
    for (int s = 0; s < LN_BWD_STAGES - 1; s++)
        fetch(first + s * step, s);
    fetch_stats(first);
    int stage = 0, buf = 0;
    size_t r0 = first;
    for (size_t base = (size_t)blockIdx.x * groups * R; base < rows; base += step, r0 += step, buf ^= 1) {
        fetch(r0 + (LN_BWD_STAGES - 1) * step, (stage + LN_BWD_STAGES - 1) % LN_BWD_STAGES);
        copy_wait<LN_BWD_STAGES - 1>();
        float s[2 * R];
#pragma unroll
        for (int k = 0; k < R; k++) {
            f32x2 a[4], g[4], s1 = 0, s2 = 0;
            unpack4x2(*at(stage, 0, k), a);
            unpack4x2(*at(stage, 1, k), g);
            const f32x2 nm = pair(-m[k], -m[k]);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const f32x2 t = mul2(g[e], wv[e]);
                s1 = add2(s1, t);
                s2 = fma2(t, add2(a[e], nm), s2);
            }
            float p, q;
            unpair(s1, p, q);
            s[2 * k] = on ? p + q : 0.f;
            unpair(s2, p, q);
            s[2 * k + 1] = on ? (p + q) * rs[k] : 0.f;
        }
        const float tot = warp_sum_many<2 * R>(s, lane);
        float* slot = sums + ((size_t)buf * groups + grp) * 2 * R * 8;
        if ((lane & (16 / R - 1)) == 0)
            slot[lane * (2 * R) / 32 * 8 + gw] = tot;
        __syncthreads();
        float c1[R], c2[R], cm[R], cr[R];
#pragma unroll
        for (int k = 0; k < R; k++) {
            const float4* t = reinterpret_cast<const float4*>(slot + 2 * k * 8);
            c1[k] = (((t[0].x + t[0].y) + (t[0].z + t[0].w)) + ((t[1].x + t[1].y) + (t[1].z + t[1].w))) * inv_d;
            c2[k] = (((t[2].x + t[2].y) + (t[2].z + t[2].w)) + ((t[3].x + t[3].y) + (t[3].z + t[3].w))) * inv_d;
            cm[k] = m[k];
            cr[k] = rs[k];
        }
        fetch_stats(r0 + step); // of the next step: used after the next wait
#pragma unroll
        for (int k = 0; k < R; k++) {
            // with x' = x - mean and the row's constants: dx = dres + rstd g - rstd c1 - (rstd^2 c2) x'
            f32x2 a[4], g[4], d[4];
            unpack4x2(*at(stage, 0, k), a);
            unpack4x2(*at(stage, 1, k), g);
            unpack4x2(dres ? *at(stage, 2, k) : make_uint4(0, 0, 0, 0), d);
            const float h0 = -cr[k] * c1[k], h1 = -cr[k] * cr[k] * c2[k];
            const f32x2 nm = pair(-cm[k], -cm[k]), r2 = pair(cr[k], cr[k]), k0 = pair(h0, h0), k1 = pair(h1, h1);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const f32x2 xc = add2(a[e], nm), gr = mul2(g[e], r2);
                acc2[0][e] = fma2(gr, xc, acc2[0][e]);
                acc2[1][e] = add2(acc2[1][e], g[e]);
                d[e] = fma2(gr, wv[e], add2(d[e], fma2(xc, k1, k0)));
            }
            if (on && r0 + k < rows) {
                const uint4 o = pack4x2(d);
                dx[(r0 + k) * packs + c] = o;
                if (COLSUM) { // of the fp32 values, before dx rounds them
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        acc2[NS - 1][e] = add2(acc2[NS - 1][e], d[e]);
                }
            }
        }
        stage = (stage + 1) % LN_BWD_STAGES;
    }
    copy_wait<0>();
    float acc[NS][8];
#pragma unroll
    for (int i = 0; i < NS; i++)
#pragma unroll
        for (int e = 0; e < 4; e++)
            unpair(acc2[i][e], acc[i][2 * e], acc[i][2 * e + 1]);
    // block partials: the groups' sums meet in shared memory in a fixed order
    const int cols = packs * 8;
    float* out = partial + (size_t)blockIdx.x * NS * cols;
    if (groups == 1) {
        if (on)
#pragma unroll
            for (int i = 0; i < NS; i++)
#pragma unroll
                for (int h = 0; h < 2; h++)
                    *reinterpret_cast<float4*>(out + (size_t)i * cols + c * 8 + h * 4) =
                        make_float4(acc[i][4 * h], acc[i][4 * h + 1], acc[i][4 * h + 2], acc[i][4 * h + 3]);
        return;
    }
#pragma unroll
    for (int i = 0; i < NS; i++) {
        __syncthreads();
        if (on)
#pragma unroll
            for (int h = 0; h < 2; h++)
                *reinterpret_cast<float4*>(sh + (size_t)grp * cols + c * 8 + h * 4) =
                    make_float4(acc[i][4 * h], acc[i][4 * h + 1], acc[i][4 * h + 2], acc[i][4 * h + 3]);
        __syncthreads();
        for (int col = threadIdx.x; col < cols; col += blockDim.x) {
            float t = 0.f;
            for (int q = 0; q < groups; q++)
                t += sh[(size_t)q * cols + col];
            out[(size_t)i * cols + col] = t;
        }
    }
}

// out[which][col] (+)= sum over `n` partial rows in a fixed order.  A block owns 32 columns of one output: 8 row groups
// add their share of the partial rows (8 loads in flight each), shared memory joins them.  grid = (cols / 32, outputs).
struct partial_outs {
    __nv_bfloat16* out[3];
    int add; // bit i: add to what output i holds
};

__global__ void __launch_bounds__(256) partial_rows_sum_kernel(const float* __restrict__ partial, int n, int cols, partial_outs o) {
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane, which = blockIdx.y;
    pdl_wait();
    float a = 0.f;
    if (c < cols) {
        const float* p = partial + (size_t)which * cols + c;
        const size_t pitch = (size_t)gridDim.y * cols;
        int k = grp;
        for (; k + 56 < n; k += 64) {
            float t[8];
#pragma unroll
            for (int i = 0; i < 8; i++)
                t[i] = __ldcg(p + (size_t)(k + 8 * i) * pitch);
#pragma unroll
            for (int i = 0; i < 8; i++)
                a += t[i];
        }
        for (; k < n; k += 8)
            a += __ldcg(p + (size_t)k * pitch);
    }
    __shared__ float sh[8][32];
    sh[grp][lane] = a;
    __syncthreads();
    if (grp == 0 && c < cols) {
        float s = 0.f;
#pragma unroll
        for (int g = 0; g < 8; g++)
            s += sh[g][lane];
        __nv_bfloat16* out = (which == 0 ? o.out[0] : which == 1 ? o.out[1] : o.out[2]) + c;
        *out = __float2bfloat16_rn(o.add >> which & 1 ? __bfloat162float(*out) + s : s);
    }
}

} // namespace

namespace {

// ---- elementwise passes over [rows, 8 * packs] that also sum their result over the rows (bias gradients) -------------
//
// Bound by memory.  A thread owns one 16-byte pack of columns and takes the rows of its block four at a time; blocks
// are short (rows_per_block) and many, in launch order, and leave one row of partial sums each, which
// partial_rows_sum_kernel adds in a fixed order.  The sum costs no pass of its own: reading the result again for it
// took 13 us per 8192 rows of 1024 to 4096 columns.
template <class F>
__global__ void __launch_bounds__(128) map_colsum_kernel(F f, size_t rows, int packs, int rows_per_block, float* __restrict__ partial) {
    const int pack = blockIdx.x * 128 + threadIdx.x;
    pdl_trigger();
    if (pack >= packs)
        return;
    const size_t r0 = (size_t)blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
    f32x2 acc[4] = { 0, 0, 0, 0 };
    for (size_t r = r0; r < r1; r += 4) {
        typename F::input in[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (r + k < r1)
                in[k] = f.load(r + k, pack);
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (r + k < r1) {
                f32x2 v[4];
                f.apply(in[k], v);
                f.store(r + k, pack, pack4x2(v));
#pragma unroll
                for (int e = 0; e < 4; e++)
                    acc[e] = add2(acc[e], v[e]);
            }
    }
    float s[8];
#pragma unroll
    for (int e = 0; e < 4; e++)
        unpair(acc[e], s[2 * e], s[2 * e + 1]);
    float4* out = reinterpret_cast<float4*>(partial + ((size_t)blockIdx.y * packs + pack) * 8);
    out[0] = make_float4(s[0], s[1], s[2], s[3]);
    out[1] = make_float4(s[4], s[5], s[6], s[7]);
}

__global__ void __launch_bounds__(256) gelu_fwd_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, size_t packs) {
    const size_t i0 = (size_t)blockIdx.x * 512 + threadIdx.x;
    uint4 u[2];
#pragma unroll
    for (int k = 0; k < 2; k++)
        if (i0 + k * 256 < packs)
            u[k] = x[i0 + k * 256];
#pragma unroll
    for (int k = 0; k < 2; k++)
        if (i0 + k * 256 < packs) {
            f32x2 v[4];
            unpack4x2(u[k], v);
#pragma unroll
            for (int e = 0; e < 4; e++)
                v[e] = mul2(v[e], gelu_gate(v[e]));
            y[i0 + k * 256] = pack4x2(v);
        }
}

// the matrix as it is: column sums alone
struct sum_map {
    const uint4* src;
    int packs;
    struct input {
        uint4 u;
    };
    __device__ __forceinline__ input load(size_t r, int p) const {
        return { src[r * packs + p] };
    }
    __device__ __forceinline__ void apply(const input& in, f32x2 (&v)[4]) const {
        unpack4x2(in.u, v);
    }
    __device__ __forceinline__ void store(size_t, int, const uint4&) const {}
};

struct gelu_bwd_map {
    const uint4 *dy, *x;
    uint4* dx;
    int packs;
    struct input {
        uint4 dy, x;
    };
    __device__ __forceinline__ input load(size_t r, int p) const {
        return { dy[r * packs + p], x[r * packs + p] };
    }
    __device__ __forceinline__ void apply(const input& in, f32x2 (&v)[4]) const {
        f32x2 a[4], g[4];
        unpack4x2(in.x, a);
        unpack4x2(in.dy, g);
#pragma unroll
        for (int e = 0; e < 4; e++)
            v[e] = mul2(g[e], gelu_slope(a[e]));
    }
    __device__ __forceinline__ void store(size_t r, int p, const uint4& u) const {
        dx[r * packs + p] = u;
    }
};

// row (b, s) of a packed QKV gradient [B, S, 3, H, dh] from three gradients with element strides of their own
struct qkv_map {
    const __nv_bfloat16* src[3];
    long long sb[3], ss[3], sh[3]; // source strides of (batch, sequence, head)
    uint4* dst;
    int S, H, ppr; // ppr: packs per head row
    struct input {
        uint4 u;
    };
    __device__ __forceinline__ input load(size_t r, int p) const {
        const int head = p / ppr, part = head / H, h = head - part * H;
        const unsigned b = (unsigned)r / (unsigned)S, s = (unsigned)r - b * (unsigned)S; // 64-bit divisions cost more than the copy
        const __nv_bfloat16* q = part == 0 ? src[0] : part == 1 ? src[1] : src[2];
        const long long o = part == 0 ? b * sb[0] + s * ss[0] + h * sh[0]
                            : part == 1 ? b * sb[1] + s * ss[1] + h * sh[1]
                                        : b * sb[2] + s * ss[2] + h * sh[2];
        return { *reinterpret_cast<const uint4*>(q + o + (p - head * ppr) * 8) };
    }
    __device__ __forceinline__ void apply(const input& in, f32x2 (&v)[4]) const {
        unpack4x2(in.u, v);
    }
    __device__ __forceinline__ void store(size_t r, int p, const uint4& u) const {
        dst[r * (size_t)(3 * H * ppr) + p] = u;
    }
};

} // namespace

// ---- C entry points -----------------------------------------------------------------------------
// D: a multiple of 8 up to 2048; 16-byte aligned rows.  mean / rstd: fp32 [rows].  res / sum_out may be null (no residual).
CCLX_API int cclx_layer_norm_fwd(const void* x, const void* res, const void* w, const void* b, void* y, void* sum_out,
                                 float* mean, float* rstd, size_t rows, int D, float eps, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(D % 8 == 0 && D >= 8 && D <= 2048, "fused LayerNorm supports multiples of 8 up to 2048 columns");
        CCL_THROW_IF_NOT((res == nullptr) == (sum_out == nullptr), "residual input and sum output go together");
        if (rows == 0)
            return;
        // four warps per block; up to 24 warps per SM, after which warps take several rows
        const int blocks = (int)std::min<size_t>((rows + 3) / 4, (size_t)device_sms() * 6);
        cudaStream_t st = (cudaStream_t)stream;
#define LN_FWD(V)                                                                                                     \
    case V:                                                                                                           \
        ln_fwd_kernel<V><<<blocks, 128, 0, st>>>((const uint4*)x, (const uint4*)res, (const uint4*)w, (const uint4*)b, \
                                                 (uint4*)y, (uint4*)sum_out, mean, rstd, rows, D / 8, 1.0f / D, eps); \
        break
        switch ((D + 255) / 256) {
            LN_FWD(1);
            LN_FWD(2);
            LN_FWD(3);
            LN_FWD(4);
            LN_FWD(5);
            LN_FWD(6);
            LN_FWD(7);
            LN_FWD(8);
        }
#undef LN_FWD
        CUDA_CHECK(cudaGetLastError());
    });
}

// rows of the backward workspace: an upper bound of the blocks that any width launches
CCLX_API int cclx_layer_norm_bwd_blocks(size_t rows) {
    return (int)std::min<size_t>(rows, (size_t)device_sms() * LN_BWD_BLOCKS);
}

namespace {
template <int R, bool COLSUM>
int launch_ln_bwd(const void* dy, const void* x, const void* w, const float* mean, const float* rstd, const void* dres,
                  void* dx, float* workspace, size_t rows, int D, cudaStream_t st) {
    const int packs = D / 8, tpr = (packs + 31) / 32 * 32;
    const int groups = std::max(1, 256 / tpr), threads = groups * tpr;
    const size_t ring = (size_t)LN_BWD_STAGES * 3 * R * threads * 16;
    const size_t smem = std::max(ring + (size_t)2 * groups * 2 * R * 8 * 4, groups > 1 ? (size_t)groups * D * 4 : 0);
    const size_t want = (rows + (size_t)groups * R - 1) / ((size_t)groups * R);
    const int blocks = (int)std::min<size_t>(want, (size_t)device_sms() * LN_BWD_BLOCKS);
    allow_smem<ln_bwd_kernel<R, COLSUM>>((size_t)LN_BWD_STAGES * 3 * R * 256 * 16 + 2048);
    ln_bwd_kernel<R, COLSUM><<<blocks, threads, smem, st>>>((const uint4*)dy, (const uint4*)x, (const uint4*)w, mean, rstd,
                                                            (const uint4*)dres, (uint4*)dx, workspace, rows, packs, tpr,
                                                            1.0f / D);
    CUDA_CHECK(cudaGetLastError());
    return blocks;
}
} // namespace

// workspace: fp32 [cclx_layer_norm_bwd_blocks(rows) * (dxsum ? 3 : 2) * D].  dres may be null.  dxsum (optional): column
// sums of dx, the bias gradient of the linear layer whose output the residual addition took.  `add`: bits 0 to 2
// say which of dgamma, dbeta and dxsum are added to what the outputs hold.  `defer` (optional) receives the number of
// partial rows in `workspace` instead: the caller sums them with cclx_partial_sums, on another stream for instance.
CCLX_API int cclx_layer_norm_bwd_sums(const void* dy, const void* x, const void* w, const float* mean, const float* rstd,
                                      const void* dres, void* dx, void* dgamma, void* dbeta, void* dxsum, int add,
                                      float* workspace, size_t rows, int D, int* defer, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(D % 8 == 0 && D >= 8 && D <= 2048, "fused LayerNorm supports multiples of 8 up to 2048 columns");
        if (rows == 0)
            return;
        cudaStream_t st = (cudaStream_t)stream;
        // Two rows per step halve the barriers; with too few rows to give every SM several steps, one row at a time
        // spreads them over the chip instead (64 rows of 1024: 32 blocks, not 16).
        const bool wide = rows >= (size_t)device_sms() * 16;
        int n;
        if (dxsum)
            n = wide ? launch_ln_bwd<LN_BWD_ROWS, true>(dy, x, w, mean, rstd, dres, dx, workspace, rows, D, st)
                     : launch_ln_bwd<1, true>(dy, x, w, mean, rstd, dres, dx, workspace, rows, D, st);
        else
            n = wide ? launch_ln_bwd<LN_BWD_ROWS, false>(dy, x, w, mean, rstd, dres, dx, workspace, rows, D, st)
                     : launch_ln_bwd<1, false>(dy, x, w, mean, rstd, dres, dx, workspace, rows, D, st);
        if (defer) {
            *defer = n;
            return;
        }
        partial_outs o{ { (__nv_bfloat16*)dgamma, (__nv_bfloat16*)dbeta, (__nv_bfloat16*)dxsum }, add };
        launch_dependent(partial_rows_sum_kernel, dim3((D + 31) / 32, dxsum ? 3 : 2), dim3(256), 0, st,
                              (const float*)workspace, n, D, o);
    });
}

namespace {
int map_rows_per_block(size_t rows, int packs) {
    // about six blocks of 128 threads per SM, between 8 and 64 rows each: fewer rows would spend more on partial sums.  More
    // only where the grid has no room for so many blocks (over 65535 of them).
    const size_t cols = (packs + 127) / 128;
    const size_t per = rows * cols / ((size_t)device_sms() * 6);
    return (int)std::max<size_t>(std::min<size_t>(64, std::max<size_t>(8, (per + 3) / 4 * 4)), (rows + 65534) / 65535);
}

template <class F>
void launch_map_colsum(const F& f, size_t rows, int packs, void* colsum, int add, float* workspace, int* defer, cudaStream_t st) {
    const int rpb = map_rows_per_block(rows, packs);
    const int n = (int)((rows + rpb - 1) / rpb);
    map_colsum_kernel<F><<<dim3((packs + 127) / 128, n), 128, 0, st>>>(f, rows, packs, rpb, workspace);
    CUDA_CHECK(cudaGetLastError());
    if (defer) {
        *defer = n;
        return;
    }
    partial_outs o{ { (__nv_bfloat16*)colsum, nullptr, nullptr }, add };
    launch_dependent(partial_rows_sum_kernel, dim3((packs * 8 + 31) / 32, 1), dim3(256), 0, st, (const float*)workspace, n,
                     packs * 8, o);
}
} // namespace

// The sums that an entry point deferred: `n` partial rows of `outputs` (1 to 3) times `cols` floats; bit i of `add`: add to
// what output i holds.
CCLX_API int cclx_partial_sums(const float* workspace, int n, int cols, int outputs, void* out0, void* out1, void* out2, int add,
                               void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(outputs >= 1 && outputs <= 3, "one to three outputs");
        partial_outs o{ { (__nv_bfloat16*)out0, (__nv_bfloat16*)out1, (__nv_bfloat16*)out2 }, add };
        partial_rows_sum_kernel<<<dim3((cols + 31) / 32, outputs), 256, 0, (cudaStream_t)stream>>>(workspace, n, cols, o);
        CUDA_CHECK(cudaGetLastError());
    });
}

// floats of workspace that the entry points below need for a result of [rows, N]
CCLX_API size_t cclx_map_colsum_workspace(size_t rows, int N) {
    const int rpb = map_rows_per_block(rows, N / 8);
    return (rows + rpb - 1) / rpb * (size_t)N;
}

// column sums of a [rows, N] bf16 matrix, added to what `out` holds if `add`
CCLX_API int cclx_colsum(const void* x, void* out, int add, float* workspace, size_t rows, int N, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(N % 8 == 0, "column count must be a multiple of 8");
        if (rows == 0 || N == 0)
            return;
        launch_map_colsum(sum_map{ (const uint4*)x, N / 8 }, rows, N / 8, out, add, workspace, nullptr, (cudaStream_t)stream);
    });
}

CCLX_API int cclx_gelu_fwd(const void* x, void* y, size_t n, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(n % 8 == 0, "the fused GELU takes whole 16-byte packs");
        if (n == 0)
            return;
        gelu_fwd_kernel<<<(unsigned)((n / 8 + 511) / 512), 256, 0, (cudaStream_t)stream>>>((const uint4*)x, (uint4*)y, n / 8);
        CUDA_CHECK(cudaGetLastError());
    });
}

// dx = dy * gelu'(x) over [rows, N], and its column sums (added to what `colsum` holds if `add`)
CCLX_API int cclx_gelu_bwd_colsum(const void* dy, const void* x, void* dx, void* colsum, int add, float* workspace, size_t rows,
                                  int N, int* defer, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(N % 8 == 0, "the fused GELU takes whole 16-byte packs");
        if (rows == 0)
            return;
        gelu_bwd_map f{ (const uint4*)dy, (const uint4*)x, (uint4*)dx, N / 8 };
        launch_map_colsum(f, rows, N / 8, colsum, add, workspace, defer, (cudaStream_t)stream);
    });
}

// packed QKV gradient out [B, S, 3, H, dh] from three [B, H, S, dh]-indexed gradients with 9 element strides (b, s, h per
// part), and its column sums
CCLX_API int cclx_qkv_grad_colsum(const void* const* src, const long long* strides, void* out, void* colsum, int add,
                                  float* workspace, int B, int S, int H, int dh, int* defer, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(dh % 8 == 0, "head size must be a multiple of 8");
        if (B == 0 || S == 0)
            return;
        CCL_THROW_IF_NOT((long long)B * S < (1ll << 31), "too many rows: ", B, " x ", S);
        qkv_map f;
        for (int p = 0; p < 3; p++) {
            f.src[p] = (const __nv_bfloat16*)src[p];
            f.sb[p] = strides[p * 3 + 0];
            f.ss[p] = strides[p * 3 + 1];
            f.sh[p] = strides[p * 3 + 2];
            CCL_THROW_IF_NOT(((uintptr_t)src[p] & 15) == 0 && f.sb[p] % 8 == 0 && f.ss[p] % 8 == 0 && f.sh[p] % 8 == 0,
                             "the QKV gradient needs 16-byte aligned rows");
        }
        f.dst = (uint4*)out;
        f.S = S;
        f.H = H;
        f.ppr = dh / 8;
        launch_map_colsum(f, (size_t)B * S, 3 * H * dh / 8, colsum, add, workspace, defer, (cudaStream_t)stream);
    });
}
