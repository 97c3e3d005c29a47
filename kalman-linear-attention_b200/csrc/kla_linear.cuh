// Linear layers of single-token decode: y[B, N] = x[B, K] W[N, K]^T for up to 64 rows of bfloat16, with what stands
// before and after the projection in a decode step folded in:
//
//   before  RMSNorm of x (src/kla/layers/common.py:45-55);
//   after   bias; the causal convolution's step on the first D outputs (common.py:87-96); silu(gate) * up
//           (common.py:99-122); the residual sum (src/kla/models/sequence_model.py:47-98).
//
// With so few rows the product is a read of W, once, from HBM or L2 (2 to 17 MB per layer and projection: 0.4 to 2.6 us
// at the measured copy rate), so the kernel is built around having enough of W in flight, not around the tensor cores:
//   * a CTA owns 16 rows of W; its eight warps take every eighth block of 32 columns and add their partial products
//     through shared memory, so that N/16 x 8 warps each have up to four 1 KB blocks of W in flight;
//   * W goes straight from global memory into the A operand of mma.m16n8k16: which column of a block a lane holds does
//     not matter to the sum as long as x is held the same way, so a lane takes 16 consecutive bytes of a row (two
//     operands' worth) instead of the four-byte pieces the operand layout names;
//   * W does not depend on the kernel before, so with programmatic dependent launch its first blocks are requested
//     before the wait for that kernel.
// Measured on B200 against the library's GEMMs, which take 4 to 5.5 us whatever the shape at these sizes:
// @@LINEAR@@
#pragma once

#include "kla_common.cuh"

namespace kla {

struct LinearParams {
    int B, N, K;
    const __nv_bfloat16 *x, *w, *bias;  // [B, K] with row stride, [N, K], [N] or nullptr
    long long x_sb, out_sb, res_sb;
    __nv_bfloat16 *out;
    const __nv_bfloat16 *norm_w;  // [K]: x is RMS-normalised first; nullptr: taken as it is
    float norm_eps;
    const __nv_bfloat16 *res;  // [B, N] added to the result, or nullptr
    // convolution step on the first D outputs (kLinearConv)
    int D, taps, conv_act;
    const float *conv_w, *conv_b;
    __nv_bfloat16 *conv_state;  // [B, D, taps-1]
};

enum LinearMode { kLinearPlain = 0, kLinearSwiglu = 1, kLinearConv = 2 };
constexpr int kLinearWarps = 8;    // warps per CTA = ways the columns are split
constexpr int kLinearMaxRows = 64;

__device__ __forceinline__ uint4 load_once(const void *p) {  // read-only, used once: not kept in L1
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 16-row tiles of W per CTA. One while x is small beside them; from 17 rows of x on two, since a CTA reads all of x for
// every tile's worth of W (at one, 32 rows: 12 us where the library takes 5). With swiglu: the gate's tile and the up's.
template <int NT, int MODE>
constexpr int kLinearTiles = MODE == kLinearSwiglu || NT >= 4 ? 2 : 1;
// blocks of W (and of x) a warp holds in flight: what the registers allow
template <int NT, int MODE>
constexpr int kLinearDepth = NT == 8 ? 2 : NT == 1 && kLinearTiles<NT, MODE> == 1 ? 8 : 4;

// shared memory: partial sums of every warp, then (NORM) the normalised rows
template <int NT, int MODE>
constexpr size_t kLinearRedBytes = sizeof(float) * kLinearWarps * kLinearTiles<NT, MODE> * 16 * (NT * 8 + 2);
inline size_t linear_norm_bytes(int nt, int K) { return sizeof(__nv_bfloat16) * nt * 8 * (K + 8); }

// RMSNorm of up to four rows at once (the warp's, W rows apart), so that their loads are in flight together. The first
// four 16-byte pieces a lane has of a row stay in registers between the two passes (K <= 1024: all of it).
template <int W, int R>
__device__ __forceinline__ void norm_rows(const LinearParams &prm, __nv_bfloat16 *xs, int xld, int r0, int lane) {
    constexpr int C = 4;
    const int chunks = prm.K / 8;
    auto at = [&](int i, int c) { return reinterpret_cast<const uint4 *>(prm.x + (long long)(r0 + i * W) * prm.x_sb + c * 8); };
    uint4 v[R][C];
    float ss[R];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j)
            v[i][j] = r0 + i * W < prm.B && lane + 32 * j < chunks ? *at(i, lane + 32 * j) : make_uint4(0, 0, 0, 0);
    auto sq = [](const uint4 &x) {
        const __nv_bfloat162 *p = reinterpret_cast<const __nv_bfloat162 *>(&x);
        float t = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(p[e]);
            t = fmaf(f.x, f.x, fmaf(f.y, f.y, t));
        }
        return t;
    };
    auto scaled = [&](uint4 x, int c, float inv) {
        const uint4 nw = *reinterpret_cast<const uint4 *>(prm.norm_w + c * 8);
        __nv_bfloat162 *p = reinterpret_cast<__nv_bfloat162 *>(&x);
        const __nv_bfloat162 *q = reinterpret_cast<const __nv_bfloat162 *>(&nw);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(p[e]), w = __bfloat1622float2(q[e]);
            p[e] = __floats2bfloat162_rn(f.x * inv * w.x, f.y * inv * w.y);
        }
        return x;
    };
#pragma unroll
    for (int i = 0; i < R; ++i) {
        ss[i] = 0.0f;
#pragma unroll
        for (int j = 0; j < C; ++j) ss[i] += sq(v[i][j]);
        if (r0 + i * W < prm.B)
            for (int c = lane + 32 * C; c < chunks; c += 32) ss[i] += sq(*at(i, c));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], o);
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (r0 + i * W >= prm.B) continue;
        const float inv = rsqrtf(ss[i] / (float)prm.K + prm.norm_eps);
        uint4 *dst = reinterpret_cast<uint4 *>(xs + (r0 + i * W) * xld);
#pragma unroll
        for (int j = 0; j < C; ++j)
            if (lane + 32 * j < chunks) dst[lane + 32 * j] = scaled(v[i][j], lane + 32 * j, inv);
        for (int c = lane + 32 * C; c < chunks; c += 32) dst[c] = scaled(*at(i, c), c, inv);
    }
}

// NT: groups of eight rows of x. MODE: LinearMode. NORM: x is normalised on the way in.
template <int NT, int MODE, bool NORM>
__global__ void __launch_bounds__(kLinearWarps * 32) kla_linear_kernel(const __grid_constant__ LinearParams prm) {
    constexpr int W = kLinearWarps, RT = kLinearTiles<NT, MODE>, U = kLinearDepth<NT, MODE>, LD = NT * 8 + 2;
    constexpr bool GLU = MODE == kLinearSwiglu;
    constexpr int ROWS = GLU ? 16 : 16 * RT;  // outputs per CTA
    extern __shared__ __align__(16) unsigned char smem[];
    float *red = reinterpret_cast<float *>(smem);  // [W][RT * 16][LD]
    __nv_bfloat16 *xs = reinterpret_cast<__nv_bfloat16 *>(smem + kLinearRedBytes<NT, MODE>);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int B = prm.B, K = prm.K, chunks = K / 8, blocks = (K + 31) / 32;
    const int n_out = GLU ? prm.N / 2 : prm.N;  // outputs per row; with swiglu W's second half is `up`
    const int row_tiles = (n_out + ROWS - 1) / ROWS;
    const int xld = K + 8;

    uint4 wl[U][RT], wh[U][RT], xv[U][NT];
    auto load_w = [&](int u, int tile, int kb) {
        const int ch = kb * 4 + t;
#pragma unroll
        for (int h = 0; h < RT; ++h) {
            const int n0 = tile * ROWS + (GLU ? 0 : h * 16) + g;
            const __nv_bfloat16 *base = prm.w + (long long)((GLU ? h * n_out : 0) + n0) * K + ch * 8;
            wl[u][h] = ch < chunks && n0 < n_out ? load_once(base) : make_uint4(0, 0, 0, 0);
            wh[u][h] = ch < chunks && n0 + 8 < n_out ? load_once(base + 8ll * K) : make_uint4(0, 0, 0, 0);
        }
    };
    auto load_x = [&](int u, int kb) {
        const int ch = kb * 4 + t;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const int r = min(nt * 8 + g, B - 1);
            xv[u][nt] = make_uint4(0, 0, 0, 0);
            if (ch < chunks) xv[u][nt] = NORM ? *reinterpret_cast<const uint4 *>(xs + r * xld + ch * 8)
                                              : *reinterpret_cast<const uint4 *>(prm.x + (long long)r * prm.x_sb + ch * 8);
        }
    };
    grid_dep_launch();
#pragma unroll
    for (int u = 0; u < U; ++u) load_w(u, blockIdx.x, warp + u * W);
    grid_dep_wait();  // everything below may read what the kernel before wrote

    if (NORM) {
        constexpr int R = NT < 4 ? NT : 4;
#pragma unroll
        for (int r0 = 0; r0 < NT; r0 += R) norm_rows<W, R>(prm, xs, xld, warp + r0 * W, lane);
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < U; ++u) load_x(u, warp + u * W);

    for (int tile = blockIdx.x; tile < row_tiles; tile += gridDim.x) {
        float acc[RT][NT][4] = {};
        for (int kb0 = warp; kb0 < blocks; kb0 += W * U) {
            const bool last = kb0 + W * U >= blocks;  // of this tile: what follows is the next tile's beginning
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int h = 0; h < RT; ++h) {
                        mma_16816(acc[h][nt], wl[u][h].x, wh[u][h].x, wl[u][h].y, wh[u][h].y, xv[u][nt].x, xv[u][nt].y);
                        mma_16816(acc[h][nt], wl[u][h].z, wh[u][h].z, wl[u][h].w, wh[u][h].w, xv[u][nt].z, xv[u][nt].w);
                    }
                // the registers just read take what comes U blocks later
                if (!last) {
                    load_w(u, tile, kb0 + (U + u) * W);
                    load_x(u, kb0 + (U + u) * W);
                } else if (tile + (int)gridDim.x < row_tiles) {
                    load_w(u, tile + gridDim.x, warp + u * W);
                    if (blocks > W * U) load_x(u, warp + u * W);  // else they are there already
                }
            }
        }
#pragma unroll
        for (int h = 0; h < RT; ++h)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
                float *dst = red + ((warp * RT + h) * 16 + g) * LD + nt * 8 + 2 * t;
                *reinterpret_cast<float2 *>(dst) = make_float2(acc[h][nt][0], acc[h][nt][1]);
                *reinterpret_cast<float2 *>(dst + 8 * LD) = make_float2(acc[h][nt][2], acc[h][nt][3]);
            }
        __syncthreads();
        for (int idx = tid; idx < ROWS * B; idx += W * 32) {
            const int i = idx % ROWS, b = idx / ROWS, n = tile * ROWS + i;
            if (n >= n_out) continue;
            auto sum = [&](int row, int bias_at) {
                float x = prm.bias != nullptr ? __bfloat162float(prm.bias[bias_at]) : 0.0f;
#pragma unroll
                for (int wp = 0; wp < W; ++wp) x += red[(wp * RT * 16 + row) * LD + b];
                return x;
            };
            float y = sum(i, n);
            if constexpr (GLU) y = activate_fast(y, kActSilu) * sum(16 + i, n_out + n);
            if constexpr (MODE == kLinearConv) {
                if (n < prm.D) {  // the window holds the projection's outputs as bfloat16
                    const int P = prm.taps - 1;
                    __nv_bfloat16 *st = prm.conv_state + ((long long)b * prm.D + n) * P;
                    const float *cw = prm.conv_w + (long long)n * prm.taps;
                    const __nv_bfloat16 xin = __float2bfloat16_rn(y);
                    float a = prm.conv_b != nullptr ? prm.conv_b[n] : 0.0f;
                    for (int j = 0; j < P; ++j) {
                        const __nv_bfloat16 old = st[j];
                        a = fmaf(cw[j], __bfloat162float(old), a);
                        if (j > 0) st[j - 1] = old;
                    }
                    a = fmaf(cw[P], __bfloat162float(xin), a);
                    if (P > 0) st[P - 1] = xin;
                    y = activate(a, prm.conv_act);
                }
            }
            if (prm.res != nullptr) y += __bfloat162float(prm.res[(long long)b * prm.res_sb + n]);
            prm.out[(long long)b * prm.out_sb + n] = __float2bfloat16_rn(y);
        }
        __syncthreads();
    }
}

}  // namespace kla
