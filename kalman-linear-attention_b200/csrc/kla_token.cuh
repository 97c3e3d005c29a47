// One decoded token through a stack of KLA blocks (or through one lone layer) as ONE persistent kernel: a CTA per SM walks
// the phases of every layer with the others,
//
//   0  [RMSNorm] in_proj + the causal convolution's step      3  [RMSNorm] w12 + silu(gate) * up
//   1  sensor_proj                                            4  w3 + residual sum
//   F  the filter step, skip path and gate                       (3, 4: blocks with a swiglu MLP)
//   2  out_proj [+ residual sum]
//
// (src/kla/layers/kla_layer.py:199-231, 277-345; src/kla/models/sequence_model.py:47-98; src/kla/layers/common.py:45-55,
// 87-122). The launcher starts it as a cooperative grid, so that all CTAs are on the chip at once.
//
// With the few rows of a token (up to eight) every phase is a read of W, and as launches of their own the phases leave HBM idle
// while each starts, waits for the one before and drains: 28 us per layer of 26 MB, 0.93 TB/s. What a phase costs here is
// latency, so there is as little of it as possible between one phase's sums and the next one's products:
//   * W waits for nobody: the whole token's weights stream, phase after phase and layer after layer, through a ring of up to
//     kTokRing stages in shared memory, ahead of the products. Every lane copies (16 bytes at a time, asynchronously) the very
//     pieces of W that it will feed to the tensor cores, into slots of its own, and asks for the next ones when it has used
//     them: no hand-over between threads, no bank conflicts. (Bulk copies of rows by one warp took it 50 cycles a copy, 1,600 a
//     stage, and everybody waited for that warp; TMA boxes of a warp's own blocks kept the TMA unit busy for 800.)
//   * there is no grid barrier. An activation travels as a 32-bit word of its bfloat16 and a 16-bit tag, and whoever needs it
//     reads it until the tag is that of this layer of this launch. A barrier costs a fence (1,150 cycles here), an atomic, a
//     poll, an acquire (900) and then the read; a tagged word costs the store and the read (below: why buffers can be reused);
//   * everything that does not depend on the phase before is fetched before its words are waited for.
// The rows of W are dealt to the CTAs in groups of eight (N = 3072 is 2.6 of them per SM: at sixteen, a third of the SMs
// would have twice the work of the others), the columns to a CTA's eight warps as in kla_linear_kernel: every sum is taken
// in the order of that kernel, norms and the filter step likewise, so that a token's results are the same to the bit.
//
// Measured on B200 in a CUDA graph, blocks of 12 layers, W from HBM, us against the separate kernels:
// d_model 768, 8 rows 270 (328), 1 row 248 (264); d_model 128, 8 rows 199 (211); d_model 1024, 4 rows 314 (354).
// What bounds it is instruction latency: 72 phases of 3.7 us, of which the words' way from CTA to CTA is 0.7; the rest is some
// 500 dependent instructions per warp. Sixteen warps take 24 % less than eight, and a spilled register costs more than it
// saves: beside this much shared memory L1 holds little.
//
// Why a buffer may be overwritten by the next layer while nothing but data says who is done: whoever reads a word in a phase has
// outputs in that phase, computed from what it read; and every output of a phase is needed, directly or through what is
// computed from it, by every output of the phase that overwrites the buffer (each phase's projections read all columns, and
// all filter outputs together read all sensor signals). So the overwriting stores come after the reads.
#pragma once

#include "kla_decode.cuh"
#include "kla_linear.cuh"

namespace kla {

constexpr int kTokWarps = 16, kTokThreads = kTokWarps * 32;
constexpr int kTokSplit = kLinearWarps;  // warps that share a tile's columns: two tiles of 16 rows of W at a time
constexpr int kTokParts = 4;             // groups of eight rows in the two tiles
constexpr int kTokCols = 512;            // columns of a stage: two blocks of 32 per warp
constexpr int kTokStage = 8 * kTokParts * kTokCols * 2;
constexpr int kTokRing = 4, kTokRingLeast = 2;  // stages of W: what fits beside x
constexpr int kTokRows = 8;              // rows of a token: one group of them in the products
constexpr int kTokLd = kTokRows + 2;     // row length of the partial sums
constexpr int kTokHeader = 256;          // of the working memory: the epoch and the number of CTAs that have left
enum TokenPhaseKind { kTokIn = 0, kTokSensor = 1, kTokOut = 2, kTokGateUp = 3, kTokDown = 4 };

// One projection: src [B, K] -> dst [B, N].
struct TokenPhase {
    const __nv_bfloat16 *w, *bias, *norm_w;  // [N, K], [N] or nullptr, [K]: x is RMS-normalised first, or nullptr
    const void *src;                         // words, or bfloat16 (plain_src)
    void *dst;                               // words, or bfloat16 (plain_dst)
    const void *res;                         // added to the result: words or bfloat16 (plain_res), or nullptr
    long long src_sb, res_sb;
    int N, K, dst_sb;    // N: outputs (of the gate half in phase 3)
    int oct_q, oct_r;    // groups of eight outputs per CTA, and how many CTAs have one more
    int plain_src, plain_dst, plain_res;
};
struct TokenLayer {
    TokenPhase ph[5];
    const float *conv_w, *conv_b;                // [M, taps], [M]; conv_w nullptr: no convolution
    __nv_bfloat16 *conv_state;                   // [B, M, taps - 1]
    const float *a, *p, *skip;                   // [M, S]; skip: nullptr, one value or [M]
    float *lam, *eta;                            // [B, M, S], updated in place
    int M, S, taps, conv_act, gate_act, gated, skip_len, w_value, qk_norm, prior, vec;
    int lpc, blocks, unit_q, unit_r;             // filter: lanes per channel, units per row, units per warp
    float obs_var_min, obs_var_max, clip;        // as StepLayerParams
    int pad;
};

template <int LAYERS>
struct TokenParams {
    int B, layers, phases, ring;  // phases: 3, with an MLP 5; stages of W
    float norm_eps;
    __nv_bfloat16 *out_var;      // [B, M] gated variance of a lone layer, or nullptr
    uint32_t *proj, *sens, *y;   // words between phases 0, 1, F, 2; rows of gated 2 M, w_value + M + 2 S, M
    unsigned *sync;
    WaitCtl wait;
    TokenLayer layer[LAYERS];
};

constexpr size_t kTokRedBytes = sizeof(float) * kTokWarps * 16 * kTokLd;  // one of two
__host__ __device__ constexpr int token_x_pitch(int K) { return (2 * K + 127) / 128 * 128 + 64; }  // bytes: four lanes read 64 bytes of a row, eight lanes of two
constexpr int kTokSmem = 226 * 1024;  // (1 KB is the kernel's own)
constexpr size_t token_smem(int widest, int ring) {
    return 2 * sizeof(TokenLayer) + ring * kTokStage + 2 * kTokRedBytes + (size_t)kTokRows * token_x_pitch(widest);
}
constexpr int token_ring(int widest) {  // 0: does not fit
    const size_t rest = token_smem(widest, 0);
    const int n = rest < kTokSmem ? (int)((kTokSmem - rest) / kTokStage) : 0;
    return n < kTokRingLeast ? 0 : n > kTokRing ? kTokRing : n;
}

__device__ __forceinline__ uint32_t ld_word(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(uint32_t *p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ uint4 ld_words(const uint32_t *p) {  // four words, each by itself current or not
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t low_halves(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5410); }
__device__ __forceinline__ uint32_t high_halves(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }
__device__ __forceinline__ float word_value(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ uint32_t make_word(float x, uint32_t tag) { return tag << 16 | __bfloat16_as_ushort(__float2bfloat16_rn(x)); }

__device__ __forceinline__ void cp_async_16_or_zero(void *dst, const void *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int LAYERS>
struct TokenCta {
    static constexpr int LD = kTokLd;
    const TokenParams<LAYERS> &prm;
    TokenLayer *ls;      // the layer at hand and the next one
    unsigned char *ring;
    float *red;          // [2][warps][16][LD]
    unsigned char *xs;   // [B] rows of x, token_x_pitch(K) bytes apart
    int *dead;           // a wait ran out: results no longer matter, nobody waits any more, all leave
    int R, stage, buf;   // stages of the ring; the next one
    int tid, lane, warp, g, t;
    // the stage of W asked for next: its layer, phase, first group of rows and first column; this lane's two rows there
    int a_layer, a_phase, a_part, a_col, a_K;
    const __nv_bfloat16 *a_lo, *a_hi;  // nullptr: not this CTA's, or past the last row

    __device__ __forceinline__ TokenCta(const TokenParams<LAYERS> &p, unsigned char *smem, int *flag)
        : prm(p), ls(reinterpret_cast<TokenLayer *>(smem)), ring(smem + 2 * sizeof(TokenLayer)), red(reinterpret_cast<float *>(ring + p.ring * kTokStage)),
          xs(ring + p.ring * kTokStage + 2 * kTokRedBytes), dead(flag), R(p.ring), stage(0), buf(0), tid(threadIdx.x),
          lane(tid & 31), warp(tid >> 5), g(lane >> 2), t(lane & 3), a_layer(0), a_phase(0), a_part(0), a_col(0) {
        static_assert(sizeof(TokenLayer) % 16 == 0, "the ring is aligned");
    }
    __device__ __forceinline__ bool gone() const { return *reinterpret_cast<volatile int *>(dead) != 0; }
    __device__ __forceinline__ void give_up(int site) {
        atomicCAS(prm.wait.status, 0, kStatusWait | site);
        *reinterpret_cast<volatile int *>(dead) = 1;
    }
    __device__ __forceinline__ void meet() { __syncthreads(); }
    __device__ __forceinline__ bool meet_and_go_on() { return !__syncthreads_or(gone()); }  // the same answer for every warp
    __device__ __forceinline__ int after(int s) const { return s + 1 == R ? 0 : s + 1; }
    // this CTA's groups of eight outputs
    __device__ __forceinline__ int octs(const TokenPhase &p) const { return p.oct_q + ((int)blockIdx.x < p.oct_r); }
    __device__ __forceinline__ int oct0(const TokenPhase &p) const { return p.oct_q * blockIdx.x + min((int)blockIdx.x, p.oct_r); }

    // ------------------------------------------------------------------------------------------------ W
    // A stage is 32 rows (two tiles of two groups of eight; in phase 3 a tile is a group of the gate's rows and one of up's) by 512
    // columns. A warp's part of it: its tile's rows, two of the sixteen blocks of columns; a lane's: 16 bytes of two rows in each.
    __device__ __forceinline__ unsigned char *slot(int s) const { return ring + s * kTokStage + warp * 2048 + lane * 16; }

    // the first pass, from (a_layer, a_phase, a_part) on, in which this CTA has rows
    __device__ __forceinline__ void enter_pass() {
#pragma unroll 1
        for (; a_layer < prm.layers;) {
            const TokenPhase &p = prm.layer[a_layer].ph[a_phase];
            const int glu = a_phase == kTokGateUp, parts = octs(p) << glu;
            if (a_part < parts) {
                const int N = p.N, part = a_part + 2 * (warp / kTokSplit), row = oct0(p) * 8 + 8 * (part >> glu) + g;
                a_K = p.K;
                const __nv_bfloat16 *w = p.w + (long long)row * a_K + ((warp % kTokSplit) * 4 + t) * 8;
                a_lo = part < parts && row < N ? w : nullptr;
                a_hi = glu ? (a_lo ? w + (long long)N * a_K : nullptr) : part + 1 < parts && row + 8 < N ? w + 8 * a_K : nullptr;
                return;
            }
            a_part = 0;
            if (++a_phase == prm.phases) {
                a_phase = 0;
                ++a_layer;
            }
        }
    }
    // Asks for the next stage of W, into slot s of the ring, which this lane has read. One group of copies per stage, empty ones
    // behind the last: the waits count groups.
    __device__ __forceinline__ void ask(int s) {
        if (a_layer < prm.layers) {
            unsigned char *dst = slot(s);
            const int col = a_col + ((warp % kTokSplit) * 4 + t) * 8;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const bool in = col + u * 256 < a_K;
                const int at = a_col + u * 256;
                cp_async_16_or_zero(dst + u * 1024, in && a_lo ? a_lo + at : prm.layer[0].ph[0].w, in && a_lo);
                cp_async_16_or_zero(dst + u * 1024 + 512, in && a_hi ? a_hi + at : prm.layer[0].ph[0].w, in && a_hi);
            }
            a_col += kTokCols;
            if (a_col >= a_K) {
                a_col = 0;
                a_part += kTokParts;
                enter_pass();
            }
        }
        cp_async_commit();
    }
    // the oldest stage is there: this lane's pieces of it
    __device__ __forceinline__ void wait_stage() {
        if (R == 4) cp_async_wait_group<3>();
        else if (R == 3) cp_async_wait_group<2>();
        else cp_async_wait_group<1>();
    }

    // What else a layer reads besides W and words, on its way from HBM to L2 while the phases in front are at work: all of it was
    // written before the launch, and most of it is read once per token. The upper warps, which have least to do, share it out.
    __device__ __forceinline__ void prefetch(const void *base, int bytes) {
        const char *at = static_cast<const char *>(base);
#pragma unroll 1
        for (int o = 128 * lane; o < bytes; o += 128 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + o));
    }
    __device__ __forceinline__ void prefetch_layer(const TokenLayer &l) {
        const int k = warp - (kTokWarps - 8);
        if (k < 0) return;
        if (k < prm.phases) {
            const TokenPhase &p = l.ph[k];
            const int n0 = oct0(p) * 8, n1 = min(n0 + 8 * octs(p), p.N);
            if (p.bias != nullptr) prefetch(p.bias + n0, 2 * (n1 - n0));
            if (p.norm_w != nullptr) prefetch(p.norm_w, 2 * p.K);
            if (k == kTokIn && l.conv_w != nullptr && n0 < l.M) {
                const int rows = min(n1, l.M) - n0, P = l.taps - 1;
                prefetch(l.conv_w + (long long)n0 * l.taps, 4 * rows * l.taps);
                if (l.conv_b != nullptr) prefetch(l.conv_b + n0, 4 * rows);
                if (lane < prm.B)
                    for (int o = 0; o < 2 * rows * P; o += 128)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char *>(l.conv_state + ((long long)lane * l.M + n0) * P) + o));
            }
        }
        if (k >= 5) {  // the filter's state, and its constants where this CTA's units stay within a row
            const int me = blockIdx.x * kTokWarps, end = me + kTokWarps, first = l.unit_q * me + min(me, l.unit_r), last = l.unit_q * end + min(end, l.unit_r);
            const int cpw = 32 / l.lpc, b0 = first / l.blocks, m0 = (first - b0 * l.blocks) * cpw;
            const long long at = ((long long)b0 * l.M + m0) * l.S, ms = (long long)m0 * l.S;
            const int n = (int)min((long long)(last - first) * cpw * l.S, (long long)prm.B * l.M * l.S - at), c = (int)min((long long)n, (long long)l.M * l.S - ms);
            if (k == 5) prefetch(l.lam + at, 4 * n);
            else if (k == 6) prefetch(l.eta + at, 4 * n);
            else {
                prefetch(l.a + ms, 4 * c);
                prefetch(l.p + ms, 4 * c);
            }
        }
    }

    // ------------------------------------------------------------------------------------------------ projections
    // The rows of x into shared memory, two warps per row, as words arrive or as they are; then normalised, a warp per row in
    // the order of kla_linear_kernel, where the phase has a norm.
    __device__ __forceinline__ void bring_x(const TokenPhase &p, uint32_t tag) {
        constexpr int U = 8;
        const int K = p.K, xp = token_x_pitch(K);
        const int r = warp >> 1;
        if (r < prm.B) {
            unsigned char *row = xs + r * xp;
            if (p.plain_src) {
                const __nv_bfloat16 *x = static_cast<const __nv_bfloat16 *>(p.src) + r * p.src_sb;
#pragma unroll 1
                for (int c = lane + 32 * (warp & 1); c < K / 8; c += 64) *reinterpret_cast<uint4 *>(row + c * 16) = __ldcg(reinterpret_cast<const uint4 *>(x + c * 8));
            } else {
#pragma unroll 1
                for (int c0 = lane * 4 + 128 * (warp & 1); c0 < K; c0 += 256 * U) {
                    const uint32_t *x = static_cast<const uint32_t *>(p.src) + r * p.src_sb + c0;
                    uint4 v[U];
                    unsigned it = 0;
                    for (;;) {
                        uint32_t off = 0;
#pragma unroll
                        for (int i = 0; i < U; ++i)
                            if (c0 + i * 256 < K) v[i] = ld_words(x + i * 256);
#pragma unroll
                        for (int i = 0; i < U; ++i)
                            if (c0 + i * 256 < K) off |= (v[i].x ^ tag << 16) | (v[i].y ^ tag << 16) | (v[i].z ^ tag << 16) | (v[i].w ^ tag << 16);
                        if (off < 0x10000u || gone()) break;
                        if (++it > prm.wait.limit_ns / 400u) {
                            give_up(41);
                            break;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < U; ++i)
                        if (c0 + i * 256 < K)
                            *reinterpret_cast<uint2 *>(row + (c0 + i * 256) * 2) = make_uint2(low_halves(v[i].x, v[i].y), low_halves(v[i].z, v[i].w));
                }
            }
        }
        if (K % 32 != 0)  // the products run over whole blocks of columns
            for (int r = warp; r < prm.B; r += kTokWarps)
                if (lane < 4 && K / 8 + lane < (K + 31) / 32 * 4) *reinterpret_cast<uint4 *>(xs + r * xp + K * 2 + lane * 16) = make_uint4(0, 0, 0, 0);
        __syncwarp();
        meet();
        if (p.norm_w != nullptr) {
            if (warp < prm.B) normalise(reinterpret_cast<uint4 *>(xs + warp * xp), p.norm_w, K);
            __syncwarp();
            meet();
        }
    }
    // norm_row, for rows of up to 1024 columns without its loops
    __device__ __forceinline__ void normalise(uint4 *row, const __nv_bfloat16 *norm_w, int K) {
        const int chunks = K / 8;
        if (chunks > 128) {
            const uint4 nw[1] = {*reinterpret_cast<const uint4 *>(norm_w + lane * 8)};
            norm_row<1>(row, nw, norm_w, chunks, K, prm.norm_eps, lane);
            return;
        }
        uint4 v[4];
        float sq[4], ss = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            v[c] = lane + 32 * c < chunks ? row[lane + 32 * c] : make_uint4(0, 0, 0, 0);
            const uint32_t w[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
            sq[c] = 0.0f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float lo = word_value(w[e]), hi = __uint_as_float(w[e] & 0xffff0000u);
                sq[c] = fmaf(lo, lo, fmaf(hi, hi, sq[c]));
            }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (lane + 32 * c < chunks) ss += sq[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        const float inv = rsqrtf(ss / (float)K + prm.norm_eps);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if (lane + 32 * c >= chunks) break;
            uint32_t w[4] = {v[c].x, v[c].y, v[c].z, v[c].w};
            const uint4 nw = *reinterpret_cast<const uint4 *>(norm_w + (lane + 32 * c) * 8);
            const uint32_t q[4] = {nw.x, nw.y, nw.z, nw.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const __nv_bfloat162 y = __floats2bfloat162_rn(word_value(w[e]) * inv * word_value(q[e]),
                                                               __uint_as_float(w[e] & 0xffff0000u) * inv * __uint_as_float(q[e] & 0xffff0000u));
                w[e] = *reinterpret_cast<const uint32_t *>(&y);
            }
            row[lane + 32 * c] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }

    // Output n of row b, number i of its pass: the warps' partial sums and what stands behind a projection.
    __device__ __forceinline__ void finish(const TokenPhase &p, const TokenLayer &l, const float *sums, bool glu, bool conv, int i, int b, int n,
                                           __nv_bfloat16 bs, __nv_bfloat16 bu, float cb, const float (&cw)[4], const __nv_bfloat16 (&cs)[3], uint32_t rs,
                                           uint32_t tag, bool silent) {
        const int P = conv ? l.taps - 1 : 0, D = l.M;
        auto sum = [&](int row, float s) {
            float x[kTokSplit];
            const float *at = sums + ((row >> 4) * kTokSplit * 16 + (row & 15)) * LD + b;
#pragma unroll
            for (int wp = 0; wp < kTokSplit; ++wp) x[wp] = at[wp * 16 * LD];
#pragma unroll
            for (int wp = 0; wp < kTokSplit; ++wp) s += x[wp];
            return s;
        };
        const int row = glu ? (i & 8) * 2 + (i & 7) : i;  // in phase 3 the gate's rows in a tile's lower half, up's in its upper
        float y = sum(row, __bfloat162float(bs));
        if (glu) y = activate_fast(y, kActSilu) * sum(row + 8, __bfloat162float(bu));
        if (conv && n < D) {  // the window holds the projection's outputs as bfloat16
            __nv_bfloat16 *st = l.conv_state + ((long long)b * D + n) * P;
            const __nv_bfloat16 xin = __float2bfloat16_rn(y);
            float a = cb, last = cw[0];
#pragma unroll
            for (int j = 0; j < 3; ++j)
                if (j < P) {
                    a = fmaf(cw[j], __bfloat162float(cs[j]), a);
                    if (j > 0) st[j - 1] = cs[j];
                    last = cw[j + 1];
                }
#pragma unroll 1
            for (int j = 3; j < P; ++j) {  // more than four taps
                const float *w = l.conv_w + (long long)n * (P + 1);
                const __nv_bfloat16 old = st[j];
                a = fmaf(w[j], __bfloat162float(old), a);
                st[j - 1] = old;
                last = w[j + 1];
            }
            a = fmaf(last, __bfloat162float(xin), a);
            if (P > 0) st[P - 1] = xin;
            y = activate(a, l.conv_act);
        }
        if (p.res != nullptr) y += word_value(rs);
        if (p.plain_dst) static_cast<__nv_bfloat16 *>(p.dst)[b * p.dst_sb + n] = __float2bfloat16_rn(y);
        else if (!silent) st_word(static_cast<uint32_t *>(p.dst) + b * p.dst_sb + n, make_word(y, tag));
    }

    // silent (test hook): the outputs are not stored
    __device__ __forceinline__ void project(const TokenLayer &l, int kind, uint32_t src_tag, uint32_t tag, bool silent) {
        const TokenPhase &p = l.ph[kind];
        const bool glu = kind == kTokGateUp, conv = kind == kTokIn && l.conv_w != nullptr;
        const int B = prm.B, N = p.N, K = p.K, parts = octs(p) << glu, first = oct0(p) * 8, xp = token_x_pitch(K), blocks = (K + 31) / 32;
        if (parts == 0) return;
        const int P = conv ? l.taps - 1 : 0, D = l.M;
        // the output of a pass that this thread finishes
        const int i = glu ? tid & 15 : lane, b = glu ? tid >> 4 : warp;
        const int kw = warp % kTokSplit;
#pragma unroll 1
        for (int part0 = 0; part0 < parts; part0 += kTokParts) {
            const int now = min(kTokParts, parts - part0), n = first + 8 * (part0 >> glu) + i;
            const bool mine = i < (8 * now >> glu) && n < N && b < B;
            // What the sums are finished with, raw, on its way while x is waited for. None of it is other CTAs' work in this launch:
            // the residual's words are this thread's own.
            uint32_t rs = 0;
            __nv_bfloat16 bs = __float2bfloat16_rn(0.0f), bu = bs, cs[3] = {bs, bs, bs};
            float cb = 0.0f, cw[4] = {};
            if (mine) {
                if (p.bias != nullptr) {
                    bs = p.bias[n];
                    if (glu) bu = p.bias[N + n];
                }
                if (p.res != nullptr) {
                    if (p.plain_res) rs = __bfloat16_as_ushort(static_cast<const __nv_bfloat16 *>(p.res)[b * p.res_sb + n]);
                    else rs = ld_word(static_cast<const uint32_t *>(p.res) + b * p.res_sb + n);
                }
                if (conv && n < D) {
                    const __nv_bfloat16 *st = l.conv_state + ((long long)b * D + n) * P;
                    const float *w = l.conv_w + (long long)n * (P + 1);
                    if (l.conv_b != nullptr) cb = l.conv_b[n];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (j < 3 && j < P) cs[j] = st[j];
                        if (j <= P) cw[j] = w[j];
                    }
                }
            }
            if (part0 == 0) bring_x(p, src_tag);
            float acc[4] = {};
            const unsigned char *x_at = xs + min(g, B - 1) * xp + kw * 64 + t * 16;
#pragma unroll 1
            for (int kb = kw; kb < blocks + kw; kb += kTokCols / 32) {
                wait_stage();
                const unsigned char *w = slot(stage);
                uint4 wl[2], wh[2], xf[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {  // (past the last column and row W is zero)
                    wl[u] = *reinterpret_cast<const uint4 *>(w + u * 1024);
                    wh[u] = *reinterpret_cast<const uint4 *>(w + u * 1024 + 512);
                    xf[u] = kb + u * kTokSplit < blocks ? *reinterpret_cast<const uint4 *>(x_at + u * 64 * kTokSplit) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    mma_16816(acc, wl[u].x, wh[u].x, wl[u].y, wh[u].y, xf[u].x, xf[u].y);
                    mma_16816(acc, wl[u].z, wh[u].z, wl[u].w, wh[u].w, xf[u].z, xf[u].w);
                }
                ask(stage);  // (the products have read the slot)
                stage = after(stage);
                x_at += 2 * kTokCols;
            }
            // partial sums of the warps; two buffers, so that one barrier per pass does
            float *sums = red + buf * (kTokRedBytes / sizeof(float));
            buf ^= 1;
            float *at = sums + (warp * 16 + g) * LD + 2 * t;
            *reinterpret_cast<float2 *>(at) = make_float2(acc[0], acc[1]);
            *reinterpret_cast<float2 *>(at + 8 * LD) = make_float2(acc[2], acc[3]);
            meet();
            if (mine) finish(p, l, sums, glu, conv, i, b, n, bs, bu, cb, cw, cs, rs, tag, silent);
        }
    }
    // ------------------------------------------------------------------------------------------------ the filter step
    // A warp's unit is 32 / lpc channels of one row, four states per lane; its state is on its way while the sensor signals' words
    // are waited for.
    __device__ __forceinline__ void filter(const TokenLayer &l, uint32_t tag) {
        const int M = l.M, S = l.S, lpc = l.lpc, blocks = l.blocks, shift = 31 - __clz(lpc), j = lane & (lpc - 1), cl = lane >> shift;
        const int me = blockIdx.x * kTokWarps + warp, first = l.unit_q * me + min(me, l.unit_r), last = first + l.unit_q + (me < l.unit_r);
        const bool vec = l.vec != 0, lane_live = j * 4 < S;
        const int p_row = (l.gated ? 2 : 1) * M, s_row = l.w_value + M + 2 * S;
        auto load4 = [&](float (&x)[4], const float *src, bool live, float pad) {
            x[0] = x[1] = x[2] = x[3] = pad;
            if (!live || !lane_live) return;
            if (vec) {
                const float4 f = *reinterpret_cast<const float4 *>(src);
                x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (j * 4 + i < S) x[i] = src[i];
            }
        };
        int b = first / blocks, block = first - b * blocks;
#pragma unroll 1
        for (int unit = first; unit < last; ++unit) {
            const int channel = block * (32 >> shift) + cl, m = min(channel, M - 1);
            const bool live = channel < M;
            const long long ms = (long long)m * S + j * 4, bms = (long long)b * M * S + ms, bm = (long long)b * M + m;
            float lamv[4], etav[4], av[4], pv[4];
            load4(lamv, l.lam + bms, live, 1.0f);
            load4(etav, l.eta + bms, live, 0.0f);
            load4(av, l.a + ms, live, 0.0f);
            load4(pv, l.p + ms, live, 1.0f);
            const float skip = l.skip != nullptr ? l.skip[l.skip_len > 1 ? m : 0] : 0.0f;
            const uint32_t *zp = prm.proj + (long long)b * p_row + m, *vp = prm.sens + (long long)b * s_row + m,
                           *kp = prm.sens + (long long)b * s_row + l.w_value + M, both = tag << 16 | tag;
            uint32_t zw, gw, vw, lw;
            uint4 kw, qw;
            unsigned it = 0;
            for (;;) {
                zw = ld_word(zp);
                gw = l.gated ? ld_word(zp + M) : zw;
                lw = ld_word(vp + l.w_value);
                vw = l.w_value ? ld_word(vp) : zw;
                if (S % 4 == 0) {
                    const int at = lane_live ? j * 4 : 0;
                    kw = ld_words(kp + at);
                    qw = ld_words(kp + S + at);
                } else {
                    auto word = [&](int e) { return ld_word(kp + min(j * 4 + e, S - 1)); };
                    auto word_q = [&](int e) { return ld_word(kp + S + min(j * 4 + e, S - 1)); };
                    kw = make_uint4(word(0), word(1), word(2), word(3));
                    qw = make_uint4(word_q(0), word_q(1), word_q(2), word_q(3));
                }
                const bool fresh = high_halves(zw, gw) == both && high_halves(lw, vw) == both && high_halves(kw.x, kw.y) == both &&
                                   high_halves(kw.z, kw.w) == both && high_halves(qw.x, qw.y) == both && high_halves(qw.z, qw.w) == both;
                if (fresh || gone()) break;
                if (++it > prm.wait.limit_ns / 400u) {
                    give_up(47);
                    break;
                }
            }
            __syncwarp();
            const uint32_t kk[4] = {kw.x, kw.y, kw.z, kw.w}, qq[4] = {qw.x, qw.y, qw.z, qw.w};
            float kv[4], qv[4], k2 = 0.0f, q2 = 0.0f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                kv[e] = j * 4 + e < S ? word_value(kk[e]) : 0.0f;
                qv[e] = j * 4 + e < S ? word_value(qq[e]) : 0.0f;
                k2 = fmaf(kv[e], kv[e], k2);
                q2 = fmaf(qv[e], qv[e], q2);
            }
            if (l.qk_norm) {  // x / max(||x||, 1e-12), src/kla/layers/common.py:25-27
                for (int off = lpc / 2; off > 0; off >>= 1) {
                    k2 += __shfl_xor_sync(0xffffffffu, k2, off);
                    q2 += __shfl_xor_sync(0xffffffffu, q2, off);
                }
                const float kn = fmaxf(sqrtf(k2), 1e-12f), qn = fmaxf(sqrtf(q2), 1e-12f);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    kv[e] /= kn;
                    qv[e] /= qn;
                }
            }
            if (l.clip > 0.0f) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    kv[e] = fminf(fmaxf(kv[e], -l.clip), l.clip);
                    qv[e] = fminf(fmaxf(qv[e], -l.clip), l.clip);
                }
            }
            const float lv = precision_from_log_variance(word_value(lw), l.obs_var_min, l.obs_var_max);
            const float vl = word_value(vw) * lv;
            float ys = 0.0f, yvs = 0.0f, lo[4], eo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float mean, var;
                filter_step(av[e], pv[e], lamv[e], etav[e], lv, vl, kv[e], l.prior != 0, lo[e], eo[e], mean, var);
                if (j * 4 + e < S) {
                    ys = fmaf(mean, qv[e], ys);
                    yvs = fmaf(var, qv[e] * qv[e], yvs);
                }
            }
            if (live && lane_live) {
                if (vec) {
                    *reinterpret_cast<float4 *>(l.lam + bms) = make_float4(lo[0], lo[1], lo[2], lo[3]);
                    *reinterpret_cast<float4 *>(l.eta + bms) = make_float4(eo[0], eo[1], eo[2], eo[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (j * 4 + e < S) {
                            l.lam[bms + e] = lo[e];
                            l.eta[bms + e] = eo[e];
                        }
                }
            }
            for (int off = lpc / 2; off > 0; off >>= 1) {
                ys += __shfl_xor_sync(0xffffffffu, ys, off);
                yvs += __shfl_xor_sync(0xffffffffu, yvs, off);
            }
            if (live && j == 0) {
                // kla_layer.py:329-338: skip path, then the gate on the mean and its square on the variance
                if (l.skip != nullptr) ys = fmaf(skip, word_value(zw), ys);
                if (l.gated) {
                    const float gt = activate(word_value(gw), l.gate_act);
                    ys *= gt;
                    yvs *= gt * gt;
                }
                st_word(prm.y + bm, make_word(ys, tag));
                if (prm.out_var != nullptr) prm.out_var[bm] = __float2bfloat16_rn(yvs);
            }
            if (++block == blocks) {
                block = 0;
                ++b;
            }
        }
    }
};

template <int LAYERS>
__global__ void __launch_bounds__(kTokThreads, 1) kla_token_kernel(const __grid_constant__ TokenParams<LAYERS> prm) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int dead;
    TokenCta<LAYERS> cta(prm, smem, &dead);
    const int tid = threadIdx.x;
    if (tid == 0) dead = 0;
    cta.enter_pass();
    for (int s = 0; s < prm.ring; ++s) cta.ask(s);
    cta.prefetch_layer(prm.layer[0]);
    const unsigned epoch = *prm.sync;  // as the launch before left it; changed when the last CTA of this one has left
    // a layer's fields from shared memory: every phase meets them for the first time, and would wait for the constant cache
    auto bring_layer = [&](int li) {
        const int at = tid - (kTokThreads - 160);  // (the upper warps have least to do)
        if (li < prm.layers && at >= 0 && at < (int)(sizeof(TokenLayer) / 4))
            reinterpret_cast<int *>(&cta.ls[li & 1])[at] = reinterpret_cast<const int *>(&prm.layer[li])[at];
    };
    static_assert(sizeof(TokenLayer) / 4 <= 160, "a thread copies a word");
    bring_layer(0);
    __syncthreads();
    int count = 0;  // phases so far, for the test hook
#pragma unroll 1
    for (int li = 0; li < prm.layers; ++li) {
        const TokenLayer &l = cta.ls[li & 1];
        const uint32_t tag = (epoch + li + 1) & 0xffff;
#pragma unroll 1
        for (int k = 0; k < prm.phases; ++k, ++count) {
            // a layer's first phase reads what the layer before left, with that layer's tag
            const uint32_t src_tag = k == kTokIn ? tag - 1 & 0xffff : tag;
            cta.project(l, k, src_tag, tag, blockIdx.x == 0 && count == prm.wait.skip_tile);
            if (k == kTokSensor) cta.filter(l, tag);
            if (k == kTokIn) bring_layer(li + 1);  // (in the slot of the layer before, which everybody has left)
            if (k == kTokOut && li + 1 < prm.layers) cta.prefetch_layer(prm.layer[li + 1]);
        }
        if (!cta.meet_and_go_on()) break;
    }
    cp_async_wait_all();
    __syncthreads();
    if (tid == 0 && atomicAdd(prm.sync + 1, 1u) == gridDim.x - 1) {
        prm.sync[0] = epoch + prm.layers;
        prm.sync[1] = 0;
    }
}

}  // namespace kla
