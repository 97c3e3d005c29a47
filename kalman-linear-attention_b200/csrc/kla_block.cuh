// What stands between a block's projections for a whole prompt (src/kla/models/sequence_model.py:47-98): the residual sum
// with the RMSNorm behind it (src/kla/layers/common.py:45-55), and the MLP's silu(gate) * up (common.py:99-122).
//
// Both are reads and writes of [rows, width] activations and bound by memory; as separate tensor operations the sum and
// norm are nine passes over them (most in float32), the gate two. One warp holds a row of the norm in registers up to a
// width of 32 x 8 x kNormPieces, so it reads x and delta once.
#pragma once

#include "kla_common.cuh"

namespace kla {

// Eight elements as 16-byte accesses (bfloat16: one, float32: two), or one by one.
template <typename T>
struct Eight {
    float x[8];
    __device__ __forceinline__ void load(const T *p) {
        if constexpr (sizeof(T) == 2) {
            const uint4 v = *reinterpret_cast<const uint4 *>(p);
            const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __bfloat1622float2(h[e]);
                x[2 * e] = f.x;
                x[2 * e + 1] = f.y;
            }
        } else {
            const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
            x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
        }
    }
    __device__ __forceinline__ void store(T *p) const {
        if constexpr (sizeof(T) == 2) {
            uint4 v;
            __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&v);
#pragma unroll
            for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(x[2 * e], x[2 * e + 1]);
            *reinterpret_cast<uint4 *>(p) = v;
        } else {
            *reinterpret_cast<float4 *>(p) = make_float4(x[0], x[1], x[2], x[3]);
            *reinterpret_cast<float4 *>(p + 4) = make_float4(x[4], x[5], x[6], x[7]);
        }
    }
};

struct AddNormParams {
    int rows, D;
    const void *x, *delta;  // [rows, D]; delta may be nullptr
    const void *w;          // [D]
    void *sum, *out;        // [rows, D]: x + delta (not written without delta), and its norm
    float eps;
};

constexpr int kNormPieces = 4;

// TW: type of the norm's weights. D is a multiple of 8 and the rows are 16-byte aligned (the host sees to it).
template <typename T, typename TW>
__global__ void __launch_bounds__(128) kla_add_norm_kernel(const __grid_constant__ AddNormParams prm) {
    const int row = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= prm.rows) return;
    const int pieces = prm.D / 8;
    const long long at = (long long)row * prm.D;
    const T *x = static_cast<const T *>(prm.x) + at, *d = prm.delta ? static_cast<const T *>(prm.delta) + at : nullptr;
    T *sum = static_cast<T *>(prm.sum) + at, *out = static_cast<T *>(prm.out) + at;
    const TW *w = static_cast<const TW *>(prm.w);
    auto take = [&](int p) {  // a piece of x + delta, rounded as it is stored
        Eight<T> v;
        v.load(x + p * 8);
        if (d != nullptr) {
            Eight<T> u;
            u.load(d + p * 8);
#pragma unroll
            for (int e = 0; e < 8; ++e) v.x[e] = to_f32<T>(from_f32<T>(v.x[e] + u.x[e]));
            v.store(sum + p * 8);
        }
        return v;
    };
    Eight<T> keep[kNormPieces];
    float ss = 0.0f;
    auto squares = [&](const Eight<T> &v) {
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(v.x[e], v.x[e], ss);
    };
#pragma unroll
    for (int j = 0; j < kNormPieces; ++j)
        if (lane + 32 * j < pieces) {
            keep[j] = take(lane + 32 * j);
            squares(keep[j]);
        }
    for (int p = lane + 32 * kNormPieces; p < pieces; p += 32) squares(take(p));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = rsqrtf(ss / (float)prm.D + prm.eps);
    auto give = [&](Eight<T> v, int p) {
        Eight<TW> nw;
        nw.load(w + p * 8);
#pragma unroll
        for (int e = 0; e < 8; ++e) v.x[e] = v.x[e] * inv * nw.x[e];
        v.store(out + p * 8);
    };
#pragma unroll
    for (int j = 0; j < kNormPieces; ++j)
        if (lane + 32 * j < pieces) give(keep[j], lane + 32 * j);
    for (int p = lane + 32 * kNormPieces; p < pieces; p += 32) {  // past the registers: this thread's own stores, or x
        Eight<T> v;
        v.load((d != nullptr ? sum : x) + p * 8);
        give(v, p);
    }
}

// The keys and queries of a prompt, l2-normalised over their states and clipped (src/kla/layers/kla_layer.py:217-222;
// common.py:25-27): one warp per (batch element, step), k in its lower and q in its upper half. As tensor operations six
// launches and 22 us at B=4 L=8192 S=16.
struct QkNormParams {
    int B, L, S;
    Tensor3 k, q;  // [B, L, S]
    void *ko, *qo; // [B, L, S] contiguous
    float clip;    // 0: none
};

template <typename T>
__global__ void __launch_bounds__(128) kla_qk_norm_kernel(const __grid_constant__ QkNormParams prm) {
    const long long row = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (row >= (long long)prm.B * prm.L) return;  // whole warps
    const int b = (int)(row / prm.L), t = (int)(row % prm.L), S = prm.S;
    const int half = (threadIdx.x >> 4) & 1, lane = threadIdx.x & 15;
    const Tensor3 &in = half ? prm.q : prm.k;
    const T *x = static_cast<const T *>(in.ptr) + (long long)b * in.sb + (long long)t * in.st;
    T *o = static_cast<T *>(half ? prm.qo : prm.ko) + row * S;
    float v[8], ss = 0.0f;  // S <= 128
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int s = lane + 16 * i;
        v[i] = s < S ? to_f32<T>(x[s]) : 0.0f;
        ss = fmaf(v[i], v[i], ss);
    }
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
    float n = sqrtf(ss);
    if (n < 1e-12f) n = 1e-12f;  // as the clamps of the tensor operations, these let a NaN through
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int s = lane + 16 * i;
        float y = v[i] / n;
        if (prm.clip > 0.0f) y = y < -prm.clip ? -prm.clip : y > prm.clip ? prm.clip : y;
        if (s < S) o[s] = from_f32<T>(y);
    }
}

// Index of the first largest value of each row (a NaN counts as the largest): a CTA per row, each thread a strided share.
// The reduction of a [8, 50304] bfloat16 head took 14 us as a tensor operation.
template <typename T>
__global__ void __launch_bounds__(1024) kla_argmax_kernel(const T *x, long long stride, int n, long long *out) {
    const T *row = x + (long long)blockIdx.x * stride;
    float best = -INFINITY;
    int at = 0x7fffffff;
    auto better = [](float v, int i, float w, int j) {  // (v, i) goes before (w, j)
        const bool nv = isnan(v), nw = isnan(w);
        if (nv != nw) return nv;
        return v > w || ((v == w || nv) && i < j);
    };
    auto see = [&](float v, int i) {
        if (better(v, i, best, at)) {
            best = v;
            at = i;
        }
    };
    const bool vec = n % 8 == 0 && stride % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    if (vec) {
        for (int p = threadIdx.x; p < n / 8; p += 1024) {
            Eight<T> v;
            v.load(row + p * 8);
#pragma unroll
            for (int e = 0; e < 8; ++e) see(v.x[e], p * 8 + e);
        }
    } else {
        for (int i = threadIdx.x; i < n; i += 1024) see(to_f32<T>(row[i]), i);
    }
    __shared__ float sv[32];
    __shared__ int si[32];
    auto warp_best = [&] {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float v = __shfl_down_sync(0xffffffffu, best, o);
            const int i = __shfl_down_sync(0xffffffffu, at, o);
            see(v, i);
        }
    };
    warp_best();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        sv[warp] = best;
        si[warp] = at;
    }
    __syncthreads();
    if (warp == 0) {
        best = sv[lane];
        at = si[lane];
        warp_best();
        if (lane == 0) out[blockIdx.x] = at;
    }
}

// out[r, i] = silu(gu[r, i]) * gu[r, H + i], eight elements per thread
template <typename T>
__global__ void __launch_bounds__(256) kla_swiglu_kernel(const T *gu, T *out, long long rows, int H) {
    const int pieces = H / 8;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= rows * pieces) return;
    const long long r = i / pieces;
    const int p = (int)(i % pieces) * 8;
    Eight<T> g, u;
    g.load(gu + r * 2 * H + p);
    u.load(gu + r * 2 * H + H + p);
#pragma unroll
    for (int e = 0; e < 8; ++e) g.x[e] = activate_fast(g.x[e], kActSilu) * u.x[e];
    g.store(out + r * H + p);
}

}  // namespace kla
