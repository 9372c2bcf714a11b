// Device kernels of the data-parallel training step that sit next to the
// gradient allreduce: squared-norm of the reduced gradient bucket, fused AdamW
// on flat buffers (fp32 master weights, bf16 model weights written in the same
// pass, gradient read in the bucket's own dtype, clipping factor taken from
// the device-resident norm), and a fused softmax cross-entropy that turns the
// bf16 logits into their gradient in place.
//
// The reference library stops at the collective; these kernels are what makes
// "allreduce fused with 1/world scale and cast" end to end: the bucket stays
// bf16 on the wire and is widened exactly once, inside the optimizer.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "capi/capi_common.hpp"
#include "core/log.hpp"
#include "gpu/async_copy.cuh"
#include "gpu/cuda_driver.hpp"
#include "gpu/f32x2.cuh"
#include "gpu/launch_util.cuh"

using namespace cclx;
using namespace cclx::gpu;

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

template <class T>
__device__ __forceinline__ float ldf(const T* p, size_t i);
template <>
__device__ __forceinline__ float ldf<float>(const float* p, size_t i) {
    return p[i];
}
template <>
__device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p, size_t i) {
    return __bfloat162float(p[i]);
}

// Squared L2 norm in two deterministic stages (every rank of a data-parallel job must get
// the same bits, otherwise the clipping factor and then the replicas drift apart):
// stage 1: block b writes sum of its grid-stride share of g^2 to partial[b];
// stage 2: one block adds the partials in a fixed tree order and accumulates into out[0].
constexpr int SQN_MAX_BLOCKS = 1024;

template <class T>
__device__ __forceinline__ float sq_pack(const uint4& u) {
    const T* h = reinterpret_cast<const T*>(&u);
    float a = 0.f;
#pragma unroll
    for (int k = 0; k < (int)(16 / sizeof(T)); k++) {
        const float v = ldf<T>(h, k);
        a = fmaf(v, v, a);
    }
    return a;
}

// Bound by memory.  A block takes pieces of SQN_PIECE 16-byte packs, eight loads in flight per thread, normally just one
// piece: blocks that loop over the buffer drift apart and lose the DRAM pages to one another (124 M bf16 gradients 51 us
// with 1024 looping blocks, 37 us with one piece per block).  With `counter` the block that finishes last adds the
// partial sums in index order, writes out[0] and re-arms the counter.
constexpr int SQN_PIECE = 8 * 512;

template <class T>
__global__ void __launch_bounds__(512) sq_norm_partial_kernel(const T* g, size_t n, float* partial, int* step_dev,
                                                              unsigned* counter, float* out) {
    constexpr size_t N = 16 / sizeof(T);
    if (step_dev && blockIdx.x == 0 && threadIdx.x == 0)
        *step_dev += 1; // read by the optimizer kernel behind this one
    const size_t nv = ((((uintptr_t)g) & 15) == 0) ? n / N : 0;
    const uint4* gv = reinterpret_cast<const uint4*>(g);
    float acc = 0.f;
    for (size_t base = (size_t)blockIdx.x * SQN_PIECE; base < nv; base += (size_t)gridDim.x * SQN_PIECE) {
        uint4 u[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const size_t i = base + k * 512 + threadIdx.x;
            u[k] = i < nv ? gv[i] : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int k = 0; k < 8; k++)
            acc += sq_pack<T>(u[k]);
    }
    for (size_t e = nv * N + (size_t)blockIdx.x * 512 + threadIdx.x; e < n; e += (size_t)gridDim.x * 512) {
        const float v = ldf<T>(g, e);
        acc = fmaf(v, v, acc);
    }
    __shared__ float part[16];
    __shared__ bool last;
    auto block_sum = [&](float v) { // in thread 0
        v = warp_sum(v);
        if ((threadIdx.x & 31) == 0)
            part[threadIdx.x >> 5] = v;
        __syncthreads();
        return threadIdx.x < 32 ? warp_sum(threadIdx.x < 16 ? part[threadIdx.x] : 0.f) : 0.f;
    };
    acc = block_sum(acc);
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = acc;
        if (counter) {
            __threadfence();
            last = atomicAdd(counter, 1u) == gridDim.x - 1;
        }
    }
    if (!counter)
        return;
    __syncthreads();
    if (last) {
        __threadfence();
        acc = 0.f;
        for (unsigned i = threadIdx.x; i < gridDim.x; i += 512)
            acc += __ldcg(partial + i);
        acc = block_sum(acc);
        if (threadIdx.x == 0) {
            out[0] = acc;
            *counter = 0;
        }
    }
}

__global__ void __launch_bounds__(SQN_MAX_BLOCKS) sq_norm_final_kernel(const float* partial, int n, float* out) {
    __shared__ float sh[SQN_MAX_BLOCKS];
    sh[threadIdx.x] = (int)threadIdx.x < n ? partial[threadIdx.x] : 0.f;
    __syncthreads();
    for (int s = SQN_MAX_BLOCKS / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s)
            sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        out[0] += sh[0];
}

__global__ void bump_step_kernel(int* step) {
    *step += 1;
}

struct adamw_args {
    float lr, beta1, beta2, eps, weight_decay;
    float bias1, bias2; // 1 - beta^t
    float grad_scale; // multiplies the gradient (1/world when the allreduce did not scale)
    float max_norm; // <= 0: no clipping
    size_t n_decay; // elements [0, n_decay) get weight decay
};

// what an element's update needs of the step, worked out once per thread
struct adamw_coef {
    float b1, b2, c1, c2, gs, eps, lr, lr_wd, ib1, ib2;
};

__device__ __forceinline__ void adamw_element(const adamw_coef& k, float g, float& p, float& m, float& v, bool decay) {
    g *= k.gs;
    m = fmaf(m, k.b1, k.c1 * g);
    v = fmaf(v, k.b2, k.c2 * g * g);
    const float upd = __fdiv_rn(m * k.ib1, sqrtf(v * k.ib2) + k.eps);
    p -= fmaf(decay ? k.lr_wd : 0.f, p, k.lr * upd);
}

// streams that are used once, in 32-byte accesses
__device__ __forceinline__ void ld_once(const float* p, float (&v)[8]) {
    asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                 : "l"(p));
}
__device__ __forceinline__ void st_once(float* p, const float (&v)[8]) {
    asm volatile("st.global.L1::no_allocate.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p),
                 "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

// One pass: read grad (T) + master/m/v (fp32), write master/m/v and the bf16 model copy.
//
// Bound by memory (28 bytes per element with bf16 gradients).  A thread takes eight elements in accesses of 16 and 32
// bytes and is done: with a grid of resident blocks that loop over the buffers the blocks drift apart and their seven
// streams scatter over the DRAM (605 us for 124 M parameters), in launch order they stay together (507 us, 6.9 TB/s).
template <class T, bool VEC>
__global__ void __launch_bounds__(128, 8)
    adamw_flat_kernel(float* __restrict__ master, const T* __restrict__ grad, float* __restrict__ m, float* __restrict__ v,
                      __nv_bfloat16* __restrict__ model, size_t n, adamw_args a, const float* __restrict__ sq_norm,
                      const int* __restrict__ step_dev) {
    pdl_wait();
    float clip = 1.f;
    if (a.max_norm > 0.f && sq_norm)
        clip = fminf(1.f, a.max_norm / (sqrtf(*sq_norm) * a.grad_scale + 1e-6f));
    if (step_dev) { // step number kept on the device: the launch can be replayed from a CUDA graph
        const float t = (float)*step_dev;
        a.bias1 = 1.f - powf(a.beta1, t);
        a.bias2 = 1.f - powf(a.beta2, t);
    }
    const adamw_coef k{ a.beta1, a.beta2, 1.f - a.beta1, 1.f - a.beta2, a.grad_scale * clip, a.eps, a.lr, a.lr * a.weight_decay,
                        1.f / a.bias1, 1.f / a.bias2 };
    const size_t gtid = (size_t)blockIdx.x * 128 + threadIdx.x;
    const size_t packs = VEC ? n / 8 : 0;
    if (gtid < packs) {
        const size_t i = gtid * 8;
        float g[8], p[8], mm[8], vv[8];
        if constexpr (sizeof(T) == 2) {
            const uint4 u = *reinterpret_cast<const uint4*>(grad + i);
            const uint32_t w[4] = { u.x, u.y, u.z, u.w };
#pragma unroll
            for (int e = 0; e < 4; e++) {
                g[2 * e] = __uint_as_float(w[e] << 16);
                g[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
            }
        }
        else {
            *reinterpret_cast<float4*>(g) = *reinterpret_cast<const float4*>(grad + i);
            *reinterpret_cast<float4*>(g + 4) = *reinterpret_cast<const float4*>(grad + i + 4);
        }
        ld_once(master + i, p);
        ld_once(m + i, mm);
        ld_once(v + i, vv);
        const long long below = (long long)a.n_decay - (long long)i; // elements of this pack that decay
#pragma unroll
        for (int e = 0; e < 8; e++)
            adamw_element(k, g[e], p[e], mm[e], vv[e], e < below);
        st_once(master + i, p);
        st_once(m + i, mm);
        st_once(v + i, vv);
        if (model) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const __nv_bfloat162 b = __floats2bfloat162_rn(p[2 * e], p[2 * e + 1]);
                w[e] = *reinterpret_cast<const uint32_t*>(&b);
            }
            *reinterpret_cast<uint4*>(model + i) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
    const size_t i = VEC ? packs * 8 + (gtid - packs) : gtid; // the last elements, or unaligned buffers
    if (gtid >= packs && i < n) {
        float p = master[i], mi = m[i], vi = v[i];
        adamw_element(k, ldf<T>(grad, i), p, mi, vi, i < a.n_decay);
        master[i] = p;
        m[i] = mi;
        v[i] = vi;
        if (model)
            model[i] = __float2bfloat16_rn(p);
    }
}

// One block per row of logits [rows, vocab] (bf16, row pitch ld).  Computes
// loss_row = logsumexp - logit[target] and overwrites the row with
// (softmax - onehot) * grad_scale, all math in fp32.  Rows whose target is
// negative (ignore) produce zero loss and zero gradient.  Columns
// [vocab, vocab + pad_cols) are alignment padding and receive zeros.
__global__ void __launch_bounds__(1024)
    softmax_xent_kernel(__nv_bfloat16* logits, const long long* targets, float* loss_rows, int vocab, size_t ld,
                        float grad_scale, int pad_cols) {
    const size_t row = blockIdx.x;
    __nv_bfloat16* x = logits + row * ld;
    const long long tgt = targets[row];
    __shared__ float red[32];
    __shared__ float s_max, s_sum;
    const int nv = vocab / 8; // whole 16-byte packs (row start is 16-byte aligned when ld % 8 == 0)
    const bool vec = (ld % 8 == 0) && ((((uintptr_t)logits) & 15) == 0);

    float mx = -INFINITY;
    if (vec) {
        const uint4* xv = reinterpret_cast<const uint4*>(x);
        for (int i = threadIdx.x; i < nv; i += blockDim.x) {
            uint4 u = xv[i];
            const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&u);
#pragma unroll
            for (int k = 0; k < 8; k++)
                mx = fmaxf(mx, __bfloat162float(h[k]));
        }
        for (int i = nv * 8 + threadIdx.x; i < vocab; i += blockDim.x)
            mx = fmaxf(mx, __bfloat162float(x[i]));
    }
    else {
        for (int i = threadIdx.x; i < vocab; i += blockDim.x)
            mx = fmaxf(mx, __bfloat162float(x[i]));
    }
    mx = warp_max(mx);
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x < 32) {
        float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : -INFINITY;
        v = warp_max(v);
        if (threadIdx.x == 0)
            s_max = v;
    }
    __syncthreads();
    mx = s_max;

    float sum = 0.f;
    if (vec) {
        const uint4* xv = reinterpret_cast<const uint4*>(x);
        for (int i = threadIdx.x; i < nv; i += blockDim.x) {
            uint4 u = xv[i];
            const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&u);
#pragma unroll
            for (int k = 0; k < 8; k++)
                sum += __expf(__bfloat162float(h[k]) - mx);
        }
        for (int i = nv * 8 + threadIdx.x; i < vocab; i += blockDim.x)
            sum += __expf(__bfloat162float(x[i]) - mx);
    }
    else {
        for (int i = threadIdx.x; i < vocab; i += blockDim.x)
            sum += __expf(__bfloat162float(x[i]) - mx);
    }
    sum = warp_sum(sum);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        red[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x < 32) {
        float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
        v = warp_sum(v);
        if (threadIdx.x == 0)
            s_sum = v;
    }
    __syncthreads();
    sum = s_sum;
    const bool ignore = tgt < 0 || tgt >= vocab;
    if (threadIdx.x == 0)
        loss_rows[row] = ignore ? 0.f : (logf(sum) + mx - __bfloat162float(x[tgt]));
    __syncthreads(); // x[tgt] is read before any thread overwrites the row
    const float inv = ignore ? 0.f : grad_scale / sum;
    // alignment padding behind the vocabulary takes no part in the softmax: zero gradient
    for (int i = vocab + threadIdx.x; i < vocab + pad_cols; i += blockDim.x)
        x[i] = __float2bfloat16_rn(0.f);
    if (vec) {
        uint4* xv = reinterpret_cast<uint4*>(x);
        for (int i = threadIdx.x; i < nv; i += blockDim.x) {
            uint4 u = xv[i];
            __nv_bfloat16* h = reinterpret_cast<__nv_bfloat16*>(&u);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                float p = __expf(__bfloat162float(h[k]) - mx) * inv;
                if ((long long)(i * 8 + k) == tgt)
                    p -= grad_scale;
                h[k] = __float2bfloat16_rn(p);
            }
            xv[i] = u;
        }
        for (int i = nv * 8 + threadIdx.x; i < vocab; i += blockDim.x) {
            float p = __expf(__bfloat162float(x[i]) - mx) * inv;
            if (i == tgt)
                p -= grad_scale;
            x[i] = __float2bfloat16_rn(p);
        }
    }
    else {
        for (int i = threadIdx.x; i < vocab; i += blockDim.x) {
            float p = __expf(__bfloat162float(x[i]) - mx) * inv;
            if (!ignore && i == tgt)
                p -= grad_scale;
            x[i] = __float2bfloat16_rn(p);
        }
    }
}

// Softmax cross-entropy kernels.  A row of logits [rows, vocab] (bf16, row pitch ld) becomes its own gradient:
// loss_row = logsumexp - logit[target], row <- (softmax - onehot) * grad_scale, all math in fp32.  Rows whose target is
// outside [0, vocab) (ignored) have zero loss and zero gradient.  Columns [vocab, vocab + pad_cols) are alignment
// padding and receive zeros.
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// largest of eight bf16 values
__device__ __forceinline__ float max8(const uint4& u) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
    const __nv_bfloat162 m = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
    return fmaxf(__low2float(m), __high2float(m));
}

// sum of 2^(x * log2(e) + shift) over eight bf16 values
__device__ __forceinline__ float exp_sum8(const uint4& u, float shift) {
    f32x2 x[4];
    unpack4x2(u, x);
    const f32x2 l2 = pair(LOG2E, LOG2E), sh = pair(shift, shift);
    float a = 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float lo, hi;
        unpair(fma2(x[i], l2, sh), lo, hi);
        a += ex2(lo) + ex2(hi);
    }
    return a;
}

// 2^(x * log2(e) + shift) * inv, minus `hit` at element `at` (0 to 7, else nowhere)
__device__ __forceinline__ uint4 grad8(const uint4& u, float shift, float inv, long long at, float hit) {
    f32x2 x[4];
    unpack4x2(u, x);
    const f32x2 l2 = pair(LOG2E, LOG2E), sh = pair(shift, shift), k = pair(inv, inv);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float lo, hi;
        unpair(fma2(x[i], l2, sh), lo, hi);
        x[i] = mul2(pair(ex2(lo), ex2(hi)), k);
    }
    if (at >= 0 && at < 8) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float lo, hi;
            unpair(x[i], lo, hi);
            x[i] = pair(at == 2 * i ? lo - hit : lo, at == 2 * i + 1 ? hi - hit : hi);
        }
    }
    return pack4x2(x);
}

// logit `at` (0 to 7) of a pack
__device__ __forceinline__ float pick8(const uint4& u, int at) {
    const uint32_t w = at < 2 ? u.x : at < 4 ? u.y : at < 6 ? u.z : u.w;
    return __uint_as_float(at & 1 ? w & 0xffff0000u : w << 16);
}

// Running maximum and sum of exponentials below it: one more pack.  The maximum rarely moves after the first packs.  Before the
// first number above -inf the sum is 0, or NaN from NaN logits, and is kept.  A share of a row may hold nothing but the type's
// lowest value (a mask), whose product with log2(e) overflows: below -1e38 exponents are taken from there and come out as 0,
// which is their part of any row that has a larger logit.
__device__ __forceinline__ float rescaled(float s, float m, float to) {
    return m == -INFINITY ? s : s * ex2((m - to) * LOG2E);
}
__device__ __forceinline__ float shift_of(float m) {
    return -fmaxf(m, -1e38f) * LOG2E;
}
__device__ __forceinline__ void online8(const uint4& u, float& m, float& shift, float& s) {
    const float pm = max8(u);
    if (pm > m) {
        s = rescaled(s, m, pm);
        m = pm;
        shift = shift_of(m);
    }
    s += exp_sum8(u, shift);
}
__device__ __forceinline__ void online1(float x, float& m, float& shift, float& s) {
    if (x > m) {
        s = rescaled(s, m, x);
        m = x;
        shift = shift_of(m);
    }
    s += ex2(fmaf(x, LOG2E, shift));
}

// Long rows.  Bound by memory (every logit read and written once) with the exponential unit close behind: two
// exponentials per logit cost 187 of the 252 us that 8192 x 50304 logits need at the copy rate.  A block keeps one
// row in shared memory.  Thread t owns packs t, t + T, ...; it copies them in with cp.async and is the only one to read
// them, so the only block-wide step per row is the exchange of (maximum, sum) pairs.  While the gradient of a row goes
// out, every pack read back is replaced at once by the same pack of the block's next row, so loads are in flight
// during stores, and the packs of a row are consumed in four groups as they arrive.  Two blocks per SM (rows up to
// 53 K logits) fill each other's gaps.  One block per row with the row in registers, which this replaces, left the
// memory idle in all phases but one: 552 us for 8192 x 50257, now 300.
template <int T>
__global__ void __launch_bounds__(T, T == 1024 ? 1 : 1024 / T)
    xent_stream_kernel(__nv_bfloat16* logits, const long long* __restrict__ targets, float* __restrict__ loss_rows, size_t rows,
                       int vocab, size_t ld, float grad_scale, int pad_cols, int ppt) {
    extern __shared__ uint4 ring[]; // [ppt][T]
    __shared__ float2 part[2][32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int nv = vocab / 8, per = (ppt + 3) / 4;
    const int tail = nv * 8 + t; // at most 7 columns behind the packs, one per thread
    pdl_trigger();
    auto fetch = [&](size_t row, int j) {
        const int i = t + j * T;
        const bool ok = row < rows && i < nv;
        copy16_async(ring + j * T + t, ok ? logits + row * ld + (size_t)i * 8 : logits, ok);
    };
    size_t row = blockIdx.x;
    for (int g = 0; g < 4; g++) {
        for (int j = g * per; j < min((g + 1) * per, ppt); j++)
            fetch(row, j);
        copy_commit();
    }
    int buf = 0;
    for (; row < rows; row += gridDim.x, buf ^= 1) {
        __nv_bfloat16* x = logits + row * ld;
        const long long tgt = targets[row];
        const float xt = tail < vocab ? __bfloat162float(x[tail]) : 0.f;
        float m = -INFINITY, shift = 0.f, s = 0.f;
        auto eat = [&](int g) {
            for (int j = g * per; j < min((g + 1) * per, ppt); j++)
                if (t + j * T < nv)
                    online8(ring[j * T + t], m, shift, s);
        };
        copy_wait<3>();
        eat(0);
        copy_wait<2>();
        eat(1);
        copy_wait<1>();
        eat(2);
        copy_wait<0>();
        eat(3);
        if (tail < vocab)
            online1(xt, m, shift, s);
        const float wm = warp_max(m);
        const float ws = warp_sum(rescaled(s, m, wm));
        if (lane == 0)
            part[buf][warp] = make_float2(wm, ws);
        __syncthreads();
        const float2 p = lane < T / 32 ? part[buf][lane] : make_float2(-INFINITY, 0.f);
        const float mx = warp_max(p.x);
        const float sum = warp_sum(rescaled(p.y, p.x, mx));
        const bool ignore = tgt < 0 || tgt >= vocab;
        const float inv = ignore ? 0.f : grad_scale / sum, hit = ignore ? 0.f : grad_scale;
        shift = -mx * LOG2E;
        if (ignore && t == 0)
            loss_rows[row] = 0.f;
        const long long at0 = ignore ? -1 : tgt;
        for (int g = 0; g < 4; g++) {
            for (int j = g * per; j < min((g + 1) * per, ppt); j++) {
                const int i = t + j * T;
                if (i < nv) {
                    const uint4 u = ring[j * T + t];
                    const long long at = at0 - (long long)i * 8;
                    if (at >= 0 && at < 8)
                        loss_rows[row] = logf(sum) + mx - pick8(u, (int)at);
                    reinterpret_cast<uint4*>(x)[i] = grad8(u, shift, inv, at, hit);
                }
                fetch(row + gridDim.x, j);
            }
            copy_commit();
        }
        if (tail < vocab) {
            float q = ex2(fmaf(xt, LOG2E, shift)) * inv;
            if (tail == at0) {
                loss_rows[row] = logf(sum) + mx - xt;
                q -= hit;
            }
            x[tail] = __float2bfloat16_rn(q);
        }
        for (int i = vocab + t; i < vocab + pad_cols; i += T)
            x[i] = __float2bfloat16_rn(0.f);
    }
    copy_wait<0>();
}

// Short rows (up to 256 * V logits): one warp per row, the row in registers, one exponential per logit, no barrier.
// A block of 1024 threads per row spent most of its time waiting for itself: 317 x 1000 took 13 us, now 3.
template <int V>
__global__ void __launch_bounds__(128)
    xent_warp_kernel(__nv_bfloat16* logits, const long long* __restrict__ targets, float* __restrict__ loss_rows, size_t rows,
                     int vocab, size_t ld, float grad_scale, int pad_cols) {
    const int lane = threadIdx.x & 31, nv = vocab / 8, tail = nv * 8 + lane;
    pdl_trigger();
    const size_t row = (size_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (row >= rows)
        return;
    __nv_bfloat16* x = logits + row * ld;
    uint4* xv = reinterpret_cast<uint4*>(x);
    const uint32_t ninf = 0xff80ff80u;
    uint4 u[V];
#pragma unroll
    for (int v = 0; v < V; v++)
        u[v] = lane + v * 32 < nv ? xv[lane + v * 32] : make_uint4(ninf, ninf, ninf, ninf);
    const long long tgt = targets[row];
    const float xt = tail < vocab ? __bfloat162float(x[tail]) : -INFINITY;
    const bool ignore = tgt < 0 || tgt >= vocab;
    float m = xt;
#pragma unroll
    for (int v = 0; v < V; v++)
        m = fmaxf(m, max8(u[v]));
    m = warp_max(m);
    const float shift = -m * LOG2E;
    float s = ex2(fmaf(xt, LOG2E, shift));
#pragma unroll
    for (int v = 0; v < V; v++)
        s += exp_sum8(u[v], shift);
    s = warp_sum(s);
    const float inv = ignore ? 0.f : grad_scale / s, hit = ignore ? 0.f : grad_scale;
    const long long at0 = ignore ? -1 : tgt;
    if (ignore && lane == 0)
        loss_rows[row] = 0.f;
#pragma unroll
    for (int v = 0; v < V; v++) {
        const int i = lane + v * 32;
        if (i < nv) {
            const long long at = at0 - (long long)i * 8;
            if (at >= 0 && at < 8)
                loss_rows[row] = logf(s) + m - pick8(u[v], (int)at);
            xv[i] = grad8(u[v], shift, inv, at, hit);
        }
    }
    if (tail < vocab) {
        float q = ex2(fmaf(xt, LOG2E, shift)) * inv;
        if (tail == at0) {
            loss_rows[row] = logf(s) + m - xt;
            q -= hit;
        }
        x[tail] = __float2bfloat16_rn(q);
    }
    for (int i = vocab + lane; i < vocab + pad_cols; i += 32)
        x[i] = __float2bfloat16_rn(0.f);
}

constexpr size_t XENT_SMEM = 226 * 1024; // shared memory of an SM that blocks can have, reserved parts aside

template <int T>
void launch_xent_stream(__nv_bfloat16* logits, const long long* targets, float* loss_rows, size_t rows, int vocab, size_t ld,
                        float grad_scale, int pad_cols, cudaStream_t st) {
    const int ppt = (vocab / 8 + T - 1) / T;
    const size_t smem = (size_t)ppt * T * 16;
    allow_smem<xent_stream_kernel<T>>(XENT_SMEM);
    const int per_sm = std::max(1, std::min((int)(XENT_SMEM / (smem + 1536)), T == 1024 ? 1 : 1024 / T));
    const int blocks = (int)std::min<size_t>(rows, (size_t)device_sms() * per_sm);
    xent_stream_kernel<T><<<blocks, T, smem, st>>>(logits, targets, loss_rows, rows, vocab, ld, grad_scale, pad_cols, ppt);
}

void launch_softmax_xent(__nv_bfloat16* logits, const long long* targets, float* loss_rows, size_t rows, int vocab,
                         size_t ld, float grad_scale, int pad_cols, cudaStream_t st) {
    const bool vec = (ld % 8 == 0) && ((((uintptr_t)logits) & 15) == 0);
    const int nv = vocab / 8;
    const unsigned warp_blocks = (unsigned)((rows + 3) / 4);
#define XENT_WARP(V) \
    xent_warp_kernel<V><<<warp_blocks, 128, 0, st>>>(logits, targets, loss_rows, rows, vocab, ld, grad_scale, pad_cols)
    // a warp's registers hold 2048 logits; longer rows stream through shared memory by a block whose threads own
    // about four to thirteen packs each, up to what the shared memory of an SM takes (106 K logits); rows that are
    // longer still or not 16-byte aligned are read three times
    if (vec && nv <= 32)
        XENT_WARP(1);
    else if (vec && nv <= 64)
        XENT_WARP(2);
    else if (vec && nv <= 128)
        XENT_WARP(4);
    else if (vec && nv <= 256)
        XENT_WARP(8);
    else if (vec && nv <= 8 * 128)
        launch_xent_stream<128>(logits, targets, loss_rows, rows, vocab, ld, grad_scale, pad_cols, st);
    else if (vec && nv <= 8 * 256)
        launch_xent_stream<256>(logits, targets, loss_rows, rows, vocab, ld, grad_scale, pad_cols, st);
    else if (vec && nv <= 13 * 512)
        launch_xent_stream<512>(logits, targets, loss_rows, rows, vocab, ld, grad_scale, pad_cols, st);
    else if (vec && nv <= 13 * 1024)
        launch_xent_stream<1024>(logits, targets, loss_rows, rows, vocab, ld, grad_scale, pad_cols, st);
    else
        softmax_xent_kernel<<<(unsigned)rows, 1024, 0, st>>>(logits, targets, loss_rows, vocab, ld, grad_scale,
                                                            pad_cols);
#undef XENT_WARP
    CUDA_CHECK(cudaGetLastError());
}

} // namespace

namespace {
size_t sq_norm_pieces(size_t n, int dt) {
    const size_t packs = n / (dt == 11 ? 8 : 4);
    return std::max<size_t>((packs + SQN_PIECE - 1) / SQN_PIECE, 1);
}

// first stage of the squared norm; returns the number of partial sums (at most `most`, a function of n alone so that
// every rank adds in the same order)
int launch_sq_norm_partials(const void* g, size_t n, int dt, float* partials, size_t most, int* step_dev, unsigned* counter,
                            float* out, cudaStream_t st) {
    CCL_THROW_IF_NOT(dt == 9 || dt == 11, "the squared norm supports float32 and bfloat16 gradients");
    const int blocks = (int)std::min(sq_norm_pieces(n, dt), most);
    if (dt == 11)
        sq_norm_partial_kernel<__nv_bfloat16><<<blocks, 512, 0, st>>>((const __nv_bfloat16*)g, n, partials, step_dev, counter, out);
    else
        sq_norm_partial_kernel<float><<<blocks, 512, 0, st>>>((const float*)g, n, partials, step_dev, counter, out);
    CUDA_CHECK(cudaGetLastError());
    return blocks;
}

template <class T>
void launch_adamw(float* master, const void* grad, float* m, float* v, void* model, size_t n, const adamw_args& a,
                  const float* sq_norm, const int* step_dev, cudaStream_t st) {
    const uintptr_t wide = (uintptr_t)master | (uintptr_t)m | (uintptr_t)v, narrow = (uintptr_t)grad | (uintptr_t)model;
    const bool vec = (wide & 31) == 0 && (narrow & 15) == 0;
    const size_t threads = vec ? n / 8 + n % 8 : n;
    launch_dependent(vec ? adamw_flat_kernel<T, true> : adamw_flat_kernel<T, false>, dim3((unsigned)((threads + 127) / 128)),
                     dim3(128), 0, st, master, (const T*)grad, m, v, (__nv_bfloat16*)model, n, a, sq_norm, step_dev);
}

void launch_adamw_any(float* master, const void* grad, int grad_dt, float* m, float* v, void* model, size_t n, const adamw_args& a,
                      const float* sq_norm, const int* step_dev, cudaStream_t st) {
    if (grad_dt == 11)
        launch_adamw<__nv_bfloat16>(master, grad, m, v, model, n, a, sq_norm, step_dev, st);
    else if (grad_dt == 9)
        launch_adamw<float>(master, grad, m, v, model, n, a, sq_norm, step_dev, st);
    else
        CCL_THROW("adamw_flat supports float32 and bfloat16 gradients");
}

adamw_args make_adamw_args(size_t n_decay, float lr, float beta1, float beta2, float eps, float weight_decay, int step,
                           float grad_scale, float max_norm) {
    return { lr, beta1, beta2, eps, weight_decay, 1.f - powf(beta1, (float)step), 1.f - powf(beta2, (float)step), grad_scale,
             max_norm, n_decay };
}
} // namespace

// dt: 9 = float32, 11 = bfloat16 (ccl datatype codes).  out[0] += sum(g^2).
// `partials`: caller-provided scratch of at least 1024 floats.
CCLX_API int cclx_sq_norm(const void* g, size_t n, int dt, float* out, float* partials, void* stream) {
    return cclx::capi::guard([&] {
        if (n == 0)
            return;
        CCL_THROW_IF_NOT(partials != nullptr, "sq_norm needs a partials buffer of 1024 floats");
        const int blocks = launch_sq_norm_partials(g, n, dt, partials, SQN_MAX_BLOCKS, nullptr, nullptr, nullptr, (cudaStream_t)stream);
        sq_norm_final_kernel<<<1, SQN_MAX_BLOCKS, 0, (cudaStream_t)stream>>>(partials, blocks, out);
        CUDA_CHECK(cudaGetLastError());
    });
}

// floats of scratch that cclx_adamw_step needs for its norm
CCLX_API size_t cclx_adamw_step_scratch(size_t n, int grad_dt) {
    return sq_norm_pieces(n, grad_dt);
}

// The whole optimizer step: squared norm of the gradient into sq_norm[0] (max_norm > 0; `counter`: a zero word that is
// zero again afterwards, one per stream of calls), the step word, and the update clipped by that norm.  step_dev (optional):
// device word holding the step number; it is advanced first and the bias corrections are taken from it instead of `step`, so
// that the launches can be replayed from a CUDA graph.
CCLX_API int cclx_adamw_step(float* master, const void* grad, int grad_dt, float* m, float* v, void* model_bf16, size_t n,
                             size_t n_decay, float lr, float beta1, float beta2, float eps, float weight_decay, int step,
                             float grad_scale, float max_norm, float* sq_norm, float* scratch, unsigned* counter,
                             int* step_dev, void* stream) {
    return cclx::capi::guard([&] {
        if (n == 0)
            return;
        cudaStream_t st = (cudaStream_t)stream;
        if (max_norm > 0.f)
            launch_sq_norm_partials(grad, n, grad_dt, scratch, SIZE_MAX, step_dev, counter, sq_norm, st);
        else if (step_dev) {
            bump_step_kernel<<<1, 1, 0, st>>>(step_dev);
            CUDA_CHECK(cudaGetLastError());
        }
        launch_adamw_any(master, grad, grad_dt, m, v, model_bf16, n,
                         make_adamw_args(n_decay, lr, beta1, beta2, eps, weight_decay, step, grad_scale, max_norm),
                         max_norm > 0.f ? sq_norm : nullptr, step_dev, st);
    });
}

namespace {
// out[0] = sum(rows[0..n)) / n, fixed summation order (one block: strided partials, warps, then the first warp)
__global__ void __launch_bounds__(1024) mean_rows_kernel(const float* rows, size_t n, float* out) {
    __shared__ float part[32];
    pdl_wait(); // launched while the kernel that fills `rows` still runs
    float acc = 0.f;
    for (size_t i = threadIdx.x; i < n; i += blockDim.x)
        acc += __ldcg(rows + i);
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        acc = warp_sum(part[threadIdx.x]);
        if (threadIdx.x == 0)
            out[0] = acc / (float)n;
    }
}
} // namespace

CCLX_API int cclx_softmax_xent(void* logits_bf16, const long long* targets, float* loss_rows, size_t rows, int vocab,
                               size_t ld, float grad_scale, int pad_cols, void* stream) {
    return cclx::capi::guard([&] {
        if (rows == 0)
            return;
        launch_softmax_xent((__nv_bfloat16*)logits_bf16, targets, loss_rows, rows, vocab, ld, grad_scale, pad_cols,
                            (cudaStream_t)stream);
    });
}

// the same with the mean of the row losses in mean_loss[0] (loss_rows: fp32 scratch [rows])
CCLX_API int cclx_softmax_xent_mean(void* logits_bf16, const long long* targets, float* loss_rows, float* mean_loss, size_t rows,
                                    int vocab, size_t ld, float grad_scale, int pad_cols, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(rows > 0, "the mean of no rows");
        launch_softmax_xent((__nv_bfloat16*)logits_bf16, targets, loss_rows, rows, vocab, ld, grad_scale, pad_cols,
                            (cudaStream_t)stream);
        launch_dependent(mean_rows_kernel, dim3(1), dim3(1024), 0, (cudaStream_t)stream, (const float*)loss_rows, rows, mean_loss);
    });
}

// ---------------------------------------------------------------------------------------------
// Mean cross-entropy without any allocation (declared and documented in gpu/xent_noalloc.h).
// The per-row losses of the regular kernel go to a fixed device array that is part of this
// library image; a one-block kernel then averages them into the caller's float.
// ---------------------------------------------------------------------------------------------
#include "gpu/xent_noalloc.h"

#include <mutex>

namespace {

// scratch: one loss per row.  Lives in every device's copy of this module until the process ends.
static __device__ __align__(256) float xent_row_scratch[CCLX_XENT_NOALLOC_MAX_ROWS];

constexpr int XENT_MAX_DEVICES = 64;
std::mutex xent_setup_mu;
float* xent_scratch_addr[XENT_MAX_DEVICES] = {};

// Device address of the scratch array on the current device.  In host code the array's name
// is only a handle for the runtime, never an address a kernel may use: ask the runtime once
// per device, with that device current.
float* xent_scratch_for_current_device() {
    int dev = -1;
    CUDA_CHECK(cudaGetDevice(&dev));
    CCL_THROW_IF_NOT(dev >= 0 && dev < XENT_MAX_DEVICES, "device index ", dev, " out of range");
    std::lock_guard<std::mutex> lk(xent_setup_mu);
    if (!xent_scratch_addr[dev]) {
        float* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress((void**)&p, xent_row_scratch);
        CCL_THROW_IF_NOT(e == cudaSuccess && p != nullptr, "cudaGetSymbolAddress(xent_row_scratch) failed: ",
                         cudaGetErrorString(e));
        xent_scratch_addr[dev] = p;
    }
    return xent_scratch_addr[dev];
}

} // namespace

CCLX_API int cclx_softmax_xent_mean_noalloc(void* logits_bf16, const long long* targets, float* mean_loss, size_t rows,
                                            int vocab, size_t ld, float grad_scale, int pad_cols, void* stream) {
    return cclx::capi::guard([&] {
        CCL_THROW_IF_NOT(rows <= (size_t)CCLX_XENT_NOALLOC_MAX_ROWS, "softmax_xent_mean_noalloc: ", rows,
                         " rows exceed the built-in scratch of ", CCLX_XENT_NOALLOC_MAX_ROWS,
                         " rows; split the batch or use cclx_softmax_xent with a caller-provided buffer");
        CCL_THROW_IF_NOT(logits_bf16 && targets && mean_loss, "softmax_xent_mean_noalloc: null pointer argument");
        CCL_THROW_IF_NOT(vocab > 0 && (size_t)(vocab + pad_cols) <= ld, "softmax_xent_mean_noalloc: bad row layout");
        if (rows == 0)
            return;
        float* scratch = xent_scratch_for_current_device();
        cudaStream_t st = (cudaStream_t)stream;
        launch_softmax_xent((__nv_bfloat16*)logits_bf16, targets, scratch, rows, vocab, ld, grad_scale, pad_cols, st);
        launch_dependent(mean_rows_kernel, dim3(1), dim3(1024), 0, st, (const float*)scratch, rows, mean_loss);
    });
}
