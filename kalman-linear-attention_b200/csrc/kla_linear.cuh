// Linear layers of single-token decode: y[B, N] = x[B, K] W[N, K]^T for up to 32 rows of bfloat16, with what stands
// before and after the projection in a decode step folded in:
//
//   before  RMSNorm of x (src/kla/layers/common.py:45-55);
//   after   bias; the causal convolution's step on the first D outputs (common.py:87-96); silu(gate) * up
//           (common.py:99-122); the residual sum (src/kla/models/sequence_model.py:47-98).
//
// With so few rows the product is a read of W, once, from HBM or L2 (2 to 17 MB per layer and projection: 0.4 to 2.6 us
// at the measured copy rate), so the kernel is built around having enough of W in flight, not around the tensor cores:
//   * a CTA owns 16 rows of W; its eight warps take every eighth block of 32 columns and add their partial products
//     through shared memory, so that N/16 x 8 warps each have up to eight 1 KB blocks of W in flight;
//   * W goes straight from global memory into the A operand of mma.m16n8k16: which column of a block a lane holds does
//     not matter to the sum as long as x is held the same way, so a lane takes 16 consecutive bytes of a row (two
//     operands' worth) instead of the four-byte pieces the operand layout names;
//   * where W does not depend on the kernel before (the caller says so), its first blocks are requested before the wait for
//     that kernel (programmatic dependent launch): all of a warp's share up to K = 2048 for up to eight rows, up to 1024 for
//     more rows and for swiglu;
// Measured on B200 in a CUDA graph, W in L2, us per projection, against the library's GEMM with what the kernel folds in as
// launches of their own:
//   B=8   3072 x 768 4.2 (4.7), with the norm 4.8 (7.2); 3104 x 1536 4.7 (6.7); 768 x 1536 3.6 (5.2); 768 x 2048 with the
//         residual 4.2 (7.2)
//   B=16  4096 x 1024 3.6 (4.2), with the norm 6.7 (7.2); 4128 x 2048 6.2 (5.2), W from HBM 5.7 (6.3); 1024 x 2048 3.8 (6.7)
//   B=32  4096 x 1024 4.8 (4.2), with the norm 10.4 (7.3); 4128 x 2048 8.3 (5.7); 1024 x 2048 5.2 (6.2)
// What bounds it is latency: about 3 us of launch, one round trip for x, the sum over warps and the store. Beyond 16 rows
// the library's kernels are the faster ones where a projection is large (kernel_pays in kla_host.cpp draws the line), but a
// call costs the host 11 us against 4, so a lone layer's token issued eagerly takes less with these (B=32 d_model 1024:
// 29 us against 41; in a graph 27.6 against 24.4, and a captured one therefore takes the library's).
#pragma once

#include "kla_common.cuh"

namespace kla {

struct LinearParams {
    int B, N, K;
    int weights_ready;  // W and norm_w may be read before the kernel in front has ended
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

// Where x is read from. Up to eight rows, and where it is normalised, from shared memory; more rows as they are straight
// into the operands, a piece beside each block of W: staging them cost every CTA 64 KB of copies before its first product
// (B=32, 4096 x 1024: 7.2 against 4.5 us).
template <int NT, bool NORM>
constexpr bool kLinearStaged = NORM || NT == 1;
// Blocks of W (and, unstaged, of x) a warp holds in flight: its share of K <= 2048, or <= 1024 where the registers allow no
// more.
template <int NT, int RT>
constexpr int kLinearDepth = NT == 1 && RT == 1 ? 8 : 4;
// shared memory: partial sums of every warp, then x (normalised with NORM)
template <int NT, int RT>
constexpr size_t kLinearRedBytes = sizeof(float) * kLinearWarps * RT * 16 * (NT * 8 + 2);
inline size_t linear_x_bytes(bool staged, int nt, int K) { return staged ? sizeof(__nv_bfloat16) * nt * 8 * (K + 8) : 0; }

__device__ __forceinline__ void cp_async_16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// RMSNorm in place of one row of x in shared memory, by one warp; nw: this lane's pieces of the norm's weights.
template <int C>
__device__ __forceinline__ void norm_row(uint4 *row, const uint4 (&nw)[C], const __nv_bfloat16 *norm_w, int chunks, int K, float eps, int lane) {
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
    float ss = 0.0f;
    for (int c = lane; c < chunks; c += 32) ss += sq(row[c]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float inv = rsqrtf(ss / (float)K + eps);
    auto scale = [&](int c, const uint4 &w4) {
        uint4 x = row[c];
        __nv_bfloat162 *p = reinterpret_cast<__nv_bfloat162 *>(&x);
        const __nv_bfloat162 *q = reinterpret_cast<const __nv_bfloat162 *>(&w4);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(p[e]), w = __bfloat1622float2(q[e]);
            p[e] = __floats2bfloat162_rn(f.x * inv * w.x, f.y * inv * w.y);
        }
        row[c] = x;
    };
#pragma unroll
    for (int j = 0; j < C; ++j)
        if (lane + 32 * j < chunks) scale(lane + 32 * j, nw[j]);
    for (int c = lane + 32 * C; c < chunks; c += 32) scale(c, *reinterpret_cast<const uint4 *>(norm_w + c * 8));
}

// NT: groups of eight rows of x. RT: 16-row tiles of W per CTA; with swiglu the gate's and the up's. NORM: x is normalised
// on the way in.
template <int NT, int RT, int MODE, bool NORM>
__global__ void __launch_bounds__(kLinearWarps * 32) kla_linear_kernel(const __grid_constant__ LinearParams prm) {
    constexpr int W = kLinearWarps, U = kLinearDepth<NT, RT>, LD = NT * 8 + 2, NW = 4;
    constexpr bool GLU = MODE == kLinearSwiglu;
    constexpr bool STAGED = kLinearStaged<NT, NORM>;
    static_assert(!GLU || RT == 2, "gate and up");
    constexpr int ROWS = GLU ? 16 : 16 * RT;  // outputs per CTA
    extern __shared__ __align__(128) unsigned char smem[];
    float *red = reinterpret_cast<float *>(smem);  // [W][RT * 16][LD]
    __nv_bfloat16 *xs = reinterpret_cast<__nv_bfloat16 *>(smem + kLinearRedBytes<NT, RT>);  // [B][K + 8]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int B = prm.B, K = prm.K, chunks = K / 8, blocks = (K + 31) / 32;
    const int n_out = GLU ? prm.N / 2 : prm.N;  // outputs per row; with swiglu W's second half is `up`
    const int row_tiles = (n_out + ROWS - 1) / ROWS;
    const int xld = K + 8;  // rows 16 bytes off a multiple of 128: the eight rows of a fragment meet different banks

    uint4 wl[U][RT], wh[U][RT], xv[STAGED ? 1 : U][NT];
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
    auto load_x = [&](uint4 (&x)[NT], int kb) {
        const int ch = kb * 4 + t;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
            const int r = min(nt * 8 + g, B - 1);
            x[nt] = make_uint4(0, 0, 0, 0);
            if (ch < chunks) x[nt] = STAGED ? *reinterpret_cast<const uint4 *>(xs + r * xld + ch * 8)
                                            : *reinterpret_cast<const uint4 *>(prm.x + (long long)r * prm.x_sb + ch * 8);
        }
    };
    if (!prm.weights_ready) grid_dep_wait();  // before the launch: the next kernel's weights are then ready too
    grid_dep_launch();
#pragma unroll
    for (int u = 0; u < U; ++u) load_w(u, blockIdx.x, warp + u * W);
    uint4 nw[NW];
    if (NORM) {
#pragma unroll
        for (int j = 0; j < NW; ++j)
            if (lane + 32 * j < chunks) nw[j] = *reinterpret_cast<const uint4 *>(prm.norm_w + (lane + 32 * j) * 8);
    }
    grid_dep_wait();  // everything below may read what the kernel before wrote

    if constexpr (STAGED) {  // all of x, one round of asynchronous copies; a warp takes whole rows
        for (int r = warp; r < B; r += W)
            for (int c = lane; c < chunks; c += 32) cp_async_16(xs + r * xld + c * 8, prm.x + (long long)r * prm.x_sb + c * 8);
        cp_async_wait_all();
        if (NORM) {
            __syncwarp();
            for (int r = warp; r < B; r += W)
                norm_row<NW>(reinterpret_cast<uint4 *>(xs + r * xld), nw, prm.norm_w, chunks, K, prm.norm_eps, lane);
        }
        __syncthreads();
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) load_x(xv[u], warp + u * W);
    }

    for (int tile = blockIdx.x; tile < row_tiles; tile += gridDim.x) {
        float acc[RT][NT][4] = {};
        for (int kb0 = warp; kb0 < blocks; kb0 += W * U) {
            const bool last = kb0 + W * U >= blocks;  // of this tile: what follows is the next tile's beginning
#pragma unroll
            for (int u = 0; u < U; ++u) {
                uint4 (&x)[NT] = xv[STAGED ? 0 : u];
                if constexpr (STAGED) load_x(x, kb0 + u * W);
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int h = 0; h < RT; ++h) {
                        mma_16816(acc[h][nt], wl[u][h].x, wh[u][h].x, wl[u][h].y, wh[u][h].y, x[nt].x, x[nt].y);
                        mma_16816(acc[h][nt], wl[u][h].z, wh[u][h].z, wl[u][h].w, wh[u][h].w, x[nt].z, x[nt].w);
                    }
                // the registers just read take what comes U blocks later
                if (!last) {
                    load_w(u, tile, kb0 + (U + u) * W);
                    if constexpr (!STAGED) load_x(x, kb0 + (U + u) * W);
                } else if (tile + (int)gridDim.x < row_tiles) {
                    load_w(u, tile + gridDim.x, warp + u * W);
                    if constexpr (!STAGED) load_x(x, warp + u * W);
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
