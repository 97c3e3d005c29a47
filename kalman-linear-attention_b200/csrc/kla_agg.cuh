// Slab / chunk aggregates: how a whole stretch of time steps acts on the filter
// state (forward) and on the backward carry (adjoint), one 32-byte record per
// chain. They are what lets the time axis be cut -- into chunks that run side by
// side on one GPU, or into slabs held by different GPUs -- because they compose
// associatively and can be folded in a few operations per cut.
//
// * forward. In homogeneous coordinates h = (x, w, z) with P = w/x and
//   mean = z/x one filter step is linear,
//       x' = (1 + p phi) x + a2 phi w,   w' = p x + a2 w,   z' = r w' + a z,
//   (the variance-form step of kla_common.cuh multiplied through by its
//   denominator), so a stretch of steps is the product of its step matrices:
//   7 numbers (m00 m01 / m10 m11 / m20 m21 m22); a common factor does not change
//   P or mean. This is the reference's trace-normalised 2x2 Moebius product
//   (src/kla/ops/kla_ops.py:76-116) extended by the row that carries the mean,
//   which lets one pass serve both recurrences instead of two dependent ones
//   (kla_ops.py:248, 274-280). The product is not formed as one. What a stretch
//   does to a state (P0, m0) is what it would do to a state known exactly at 0,
//   the filter itself run from (C, b) = (0, 0), and how the knowledge of m0 that
//   the stretch's observations carry changes that:
//       P = C + A^2 P0 / (1 + J P0),   mean = b + A (m0 + eta P0) / (1 + J P0),
//   with A' = a A g, J' = J + phi (a A) A', eta' = eta + A' (r - phi a b), g the
//   gain of the run from 0. That is 15 pair operations a step where the matrices
//   take 18.5 with their rescaling, five numbers that stay in range by themselves,
//   and the record is (1, J / C, C J + A^2 / b, b J + A eta, A) over 1 + J.
//
// * adjoint. With the forward trajectory fixed, the backward carries obey
//   c_{t-1} = J_t (c_t + e_t), J_t = [[a2 g^2, a2 g (r - phi mean_t)], [0, a g]],
//   e_t = (dyvar q^2, dy q): affine, upper triangular. Walking FORWARD in time,
//   K_t = J_1 ... J_t and b = sum_t K_t e_t give the carry that leaves the
//   stretch at its first step as K c_in + b (5 numbers). It needs the stretch's
//   true initial state, i.e. it runs after the forward fold. With a2 = a^2 and
//   r - phi mean_t = g (r - phi a mean_{t-1}) the diagonal is one product,
//   K00 = K11^2, and K01 = K11 R with R' = R + K11' (r - phi a mean): 19 pair
//   operations a step instead of 25.
//
// Both forms take a2 for a^2, which it is but for its floor of 1e-12, binding where |a| < 1e-6. A chain that the floor binds
// forgets what came before within a few steps, 1e-6 a step at least, so the floor shows in the records of stretches of a few steps
// and in the first terms of b0. Stretches of up to kAggFloorSteps steps are composed with it by kla_agg_short_kernel (forward),
// and the adjoint walks that many steps of such a chain once more.
//
// Both walks keep -a, -a2 and -p as their constants and -Pp, -1/d as they go:
// every product then has the sign the next sum needs, since a pair instruction
// has no operand negation.
//
// Kernel shape: as the scan kernels. NW compute warps, each thread owning SPT
// states of one channel as pairs (paired fp32 instructions), and one loader warp
// that brings tiles of TT steps in: v, lambda_v (and dy, dy_var) as TMA tiles
// signalled on mbarriers, k (and q) regrouped by owning lane. Nothing is written but the final record.
// Measured on B200, B=2 L=1024 M=1024 S=16 in 4 chunks, float32, against the form with matrices: forward 29.7 -> 26.7 us,
// adjoint 39.8 -> 33.7; 192 CTAs of eight tiles: bound by the FP32 pipe of the 44 SMs that hold two (17.7 of the forward's time)
// and by the latency of the first and last tile. In 8 chunks of 512 steps (L=4096, 448 CTAs) 94 and 119 us.
#pragma once

#include "kla_common.cuh"

namespace kla {

constexpr int kAggStages = 3;
constexpr int kAggTT = 32;  // steps per tile
constexpr int kAggFloorSteps = 8;  // after which 1e-6 a step leaves less than float32 holds

struct alignas(64) AggParams {
    CUtensorMap tm_v, tm_lv, tm_dy, tm_dyv;  // rank-3 (M, L, B) maps with box (MC, kAggTT, 1); valid when use_tma
    int B, L, M, S;
    int use_tma;
    Tensor3 v, lv, k, q, dy, dyv;      // dy, dyv, q: adjoint only
    const float *a, *p, *lam0, *eta0;  // lam0/eta0: adjoint only (nullptr = unit prior)
    float *out;                        // [entries, M, S, 8]
    // lv holds log-variances, as in FwdParams: every warp turns its channels of a tile into precisions, into kLam bytes behind
    // the stages (one buffer: a warp is done with a tile before it meets the next)
    int lv_log_sigma;
    float obs_var_min, obs_var_max;
    ChunkCtl chunk;
    WaitCtl wait;
};

template <typename T, typename TO, int SPT, int LPC, int NW, bool ADJ>
struct AggSmem {
    static constexpr int kMC = NW * (32 / LPC);
    static constexpr int kSPad = SPT * LPC;
    static constexpr size_t kBars = 128;
    static constexpr size_t kTileI = ((sizeof(T) * kAggTT * kMC + 127) / 128) * 128;
    static constexpr size_t kTileO = ((sizeof(TO) * kAggTT * kMC + 127) / 128) * 128;
    static constexpr size_t kKq = ((sizeof(float) * (ADJ ? 2 : 1) * kAggTT * kSPad + 127) / 128) * 128;
    static constexpr size_t kIn = 2 * kTileI + (ADJ ? 2 * kTileO : 0) + kKq;
    static constexpr size_t kTotal = kBars + kAggStages * kIn;
    static constexpr size_t kLam = sizeof(float) * kAggTT * kMC;
};

// The first steps of a stretch of L steps from t_off on, one chain, with the floor of a2: the adjoint's five sums, which with the
// run from (0, 0) are also how the forward's posterior depends on P0 and m0 (K00 in place of A^2, K01 in place of A eta). Writes
// the record of a stretch that these are all steps of, or adds to the adjoint's b0 what the form without the floor left out.
template <typename T, typename TO, bool ADJ, bool PRIOR, bool LOGV>
__device__ __forceinline__ void walk_with_floor(const AggParams &prm, int be, int b, int t_off, int L, int m, int s, float a) {
    const long long ms = (long long)m * prm.S + s, at = (long long)be * prm.M * prm.S + ms;
    const float a2 = fmaxf(a * a, kEps), p = fmaxf(prm.p[ms], kPMin);
    float P = 0.0f, mean = 0.0f;
    if (ADJ) {
        P = prm.lam0 != nullptr ? 1.0f / fmaxf(prm.lam0[at], kLamMin) : 1.0f;
        if (prm.lam0 != nullptr) mean = prm.eta0[at] * P;
    }
    float K00 = 1.0f, K01 = 0.0f, K11 = 1.0f, R = 0.0f, J = 0.0f, b0 = 0.0f, b1 = 0.0f, missed = 0.0f;
    const int n = min(L, kAggFloorSteps);
#pragma unroll 1
    for (int tt = 0; tt < n; ++tt) {
        auto load = [&](const Tensor3 &x, int column) { return (long long)b * x.sb + (long long)(t_off + tt) * x.st + column; };
        float lv = to_f32<T>(static_cast<const T *>(prm.lv.ptr)[load(prm.lv, m)]);
        if (LOGV) lv = precision_from_log_variance_fast(lv, prm.obs_var_min, prm.obs_var_max);
        const float v = to_f32<T>(static_cast<const T *>(prm.v.ptr)[load(prm.v, m)]), k = to_f32<T>(static_cast<const T *>(prm.k.ptr)[load(prm.k, s)]);
        const float phi = lv * k * k, r = v * (lv * k);
        const float Pp = fmaf(a2, P, p), g = 1.0f / fmaf(phi, Pp, 1.0f), t = fmaf(-phi, a * mean, r);
        J = fmaf(phi * a2, K00 * g, J);
        K00 *= a2 * g * g;
        K01 = fmaf(K00, t, K01 * (a * g));
        K11 *= a * g;
        P = Pp * g;
        mean = g * fmaf(Pp, r, a * mean);
        if constexpr (ADJ) {
            const float q = to_f32<T>(static_cast<const T *>(prm.q.ptr)[load(prm.q, s)]);
            float e0 = 0.0f, e1 = to_f32<TO>(static_cast<const TO *>(prm.dy.ptr)[load(prm.dy, m)]) * q;
            if (prm.dyv.ptr != nullptr) e0 = to_f32<TO>(static_cast<const TO *>(prm.dyv.ptr)[load(prm.dyv, m)]) * q * q;
            if (PRIOR) e1 *= a;
            R = fmaf(K11, t, R);
            b0 += K00 * (PRIOR ? a2 : 1.0f) * e0 + K01 * e1;
            b1 = fmaf(K11, e1, b1);
            missed += (K00 * (PRIOR ? a2 : 1.0f) - K11 * K11 * (PRIOR ? a * a : 1.0f)) * e0 + (K01 - K11 * R) * e1;
        }
    }
    float4 *o = reinterpret_cast<float4 *>(prm.out + at * 8);
    if constexpr (ADJ) {
        if (L > n) {
            prm.out[at * 8 + 3] += missed;
            return;
        }
        o[0] = make_float4(K00, K01, K11, b0);
        o[1] = make_float4(b1, P, mean, 0.0f);
    } else {
        const float sc = 1.0f / (1.0f + J);
        o[0] = make_float4(sc, J * sc, P * sc, fmaf(P, J, K00) * sc);
        o[1] = make_float4(mean * sc, fmaf(mean, J, K01) * sc, K11 * sc, 0.0f);
    }
}

// Forward records of stretches of up to kAggFloorSteps steps, a thread per chain.
template <typename T, bool LOGV>
__global__ void __launch_bounds__(128) kla_agg_short_kernel(const __grid_constant__ AggParams prm) {
    const long long lanes = (long long)prm.M * prm.S, gid = (long long)blockIdx.x * 128 + threadIdx.x;
    if (gid >= prm.B * lanes) return;
    const int be = (int)(gid / lanes);
    const long long ms = gid % lanes;
    const ChunkSpan span = chunk_span(prm.chunk, be, prm.L);
    if (prm.chunk.n > 1 && be % prm.chunk.n == prm.chunk.n - 1) return;  // as kla_agg_kernel
    walk_with_floor<T, float, false, false, LOGV>(prm, be, span.b, span.t_off, span.L, (int)(ms / prm.S), (int)(ms % prm.S), prm.a[ms]);
}

// LOGV (AggParams::lv_log_sigma) is a separate instantiation: a test in every step cost plain inference at B=1 L=1501
// M=1536 float32 2 of its 64 us.
template <typename T, typename TO, int SPT, int LPC, int NW, bool ADJ, bool PRIOR, bool LOGV>
__global__ void __launch_bounds__((NW + 1) * 32) kla_agg_kernel(const __grid_constant__ AggParams prm) {
    using Sm = AggSmem<T, TO, SPT, LPC, NW, ADJ>;
    constexpr int TT = kAggTT, NS = kAggStages, MC = Sm::kMC, SPAD = Sm::kSPad, CLS = 32 / LPC;
    constexpr int HP = SPT / 2, NK = ADJ ? 2 : 1;
    static_assert(SPT % 2 == 0, "states are processed in pairs");
    constexpr int kCompute = NW * 32;

    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *full_in = reinterpret_cast<uint64_t *>(smem);  // [NS] loader -> compute
    uint64_t *empty_in = full_in + NS;                       // [NS] compute -> loader
    unsigned char *in_base = smem + Sm::kBars;
    auto vstage = [&](int s) { return reinterpret_cast<T *>(in_base + s * Sm::kIn); };
    auto lstage = [&](int s) { return reinterpret_cast<T *>(in_base + s * Sm::kIn + Sm::kTileI); };
    auto dystage = [&](int s) { return reinterpret_cast<TO *>(in_base + s * Sm::kIn + 2 * Sm::kTileI); };
    auto dyvstage = [&](int s) { return reinterpret_cast<TO *>(in_base + s * Sm::kIn + 2 * Sm::kTileI + Sm::kTileO); };
    // k (and q) of a step, grouped by owning lane: [TT][NK][LPC][SPT] floats, state s = i * LPC + j at [.][j][i]
    auto kqstage = [&](int s) {
        return reinterpret_cast<float *>(in_base + s * Sm::kIn + 2 * Sm::kTileI + (ADJ ? 2 * Sm::kTileO : 0));
    };

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int be = blockIdx.y, m_cta = blockIdx.x * MC;  // be: batch entry, what states and records are indexed by
    const ChunkSpan span = chunk_span(prm.chunk, be, prm.L);
    const int b = span.b, t_off = span.t_off, L = span.L, M = prm.M, S = prm.S;
    // no fold reads how the last chunk acts on the state, nor how the first acts on the carry
    if (prm.chunk.n > 1 && be % prm.chunk.n == (ADJ ? 0 : prm.chunk.n - 1)) return;
    const int NT = (L + TT - 1) / TT;
    const bool has_dyv = ADJ && prm.dyv.ptr != nullptr;
    float *lam_tile = reinterpret_cast<float *>(smem + Sm::kTotal);  // [TT][MC], with LOGV

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(&full_in[s], stage_arrivals(prm.use_tma, 32));
            mbar_init(&empty_in[s], NW);
        }
        mbar_fence_init();
    }
    __syncthreads();

    if (warp < NW) {
        // =============================================================== compute
        const int j = lane % LPC, cl = lane / LPC;
        const int cw = warp * CLS + cl;  // this thread's channel, CTA-relative
        const int m = m_cta + cw;
        float2 na[HP], na2[HP], np[HP];  // negated constants
        // forward: A, b, C, -J, eta; adjoint: K11, R, b0, b1, P, mean
        constexpr int NA = ADJ ? 6 : 5;
        float2 A[NA][HP];
#pragma unroll
        for (int i = 0; i < SPT; ++i) {
            const int s = i * LPC + j;
            const bool live = (m < M) && (s < S);
            const float av = live ? prm.a[(long long)m * S + s] : 0.0f;
            const float pv = live ? prm.p[(long long)m * S + s] : 1.0f;
            pair_el(na, i) = -av;
            pair_el(na2, i) = live ? -fmaxf(av * av, kEps) : 0.0f;
            pair_el(np, i) = -fmaxf(pv, kPMin);
            pair_el(A[0], i) = 1.0f;
#pragma unroll
            for (int e = 1; e < NA; ++e) pair_el(A[e], i) = 0.0f;
            if (ADJ) {
                float lam = 1.0f, eta = 0.0f;
                if (live && prm.lam0 != nullptr) {
                    lam = prm.lam0[((long long)be * M + m) * S + s];
                    eta = prm.eta0[((long long)be * M + m) * S + s];
                }
                const float P0 = 1.0f / fmaxf(lam, kLamMin);
                pair_el(A[NA - 2], i) = P0;
                pair_el(A[NA - 1], i) = eta * P0;
            }
        }

        auto step = [&](const T *vrow, const T *lrow, const TO *dyrow, const TO *dyvrow, const float *kqrow, int tt) {
            const float2 lv = dup2(LOGV ? lam_tile[tt * MC + cw] : to_f32<T>(lrow[tt * MC])), vv = dup2(to_f32<T>(vrow[tt * MC]));
            const float *row = kqrow + tt * NK * SPAD;
            float2 kk[HP], qq[HP];
            if constexpr (SPT == 4) {
                const float4 k4 = *reinterpret_cast<const float4 *>(row);
                kk[0] = make_float2(k4.x, k4.y);
                kk[1] = make_float2(k4.z, k4.w);
                if (ADJ) {
                    const float4 q4 = *reinterpret_cast<const float4 *>(row + SPAD);
                    qq[0] = make_float2(q4.x, q4.y);
                    qq[1] = make_float2(q4.z, q4.w);
                }
            } else {
#pragma unroll
                for (int h = 0; h < HP; ++h) {
                    kk[h] = *reinterpret_cast<const float2 *>(row + 2 * h);
                    if (ADJ) qq[h] = *reinterpret_cast<const float2 *>(row + SPAD + 2 * h);
                }
            }
            float dyf = 0.0f, dyvf = 0.0f;
            if constexpr (ADJ) {
                dyf = to_f32<TO>(dyrow[tt * MC]);
                dyvf = to_f32<TO>(dyvrow[tt * MC]);
            }
            constexpr int iP = ADJ ? 4 : 2, iM = ADJ ? 5 : 1;  // variance and mean of the run
            float2 nPp[HP], ng[HP], r[HP], phi[HP];
#pragma unroll
            for (int h = 0; h < HP; ++h) {
                chain_inputs2(lv, vv, kk[h], phi[h], r[h]);
                nPp[h] = fma2(na2[h], A[iP][h], np[h]);
                ng[h] = fma2(phi[h], nPp[h], make_float2(-1.0f, -1.0f));
            }
#pragma unroll
            for (int h = 0; h < HP; ++h) ng[h] = rcp_approx2(ng[h]);
#pragma unroll
            for (int h = 0; h < HP; ++h) {
                const float2 nam = mul2(na[h], A[iM][h]), t = fma2(phi[h], nam, r[h]), naA = mul2(na[h], A[0][h]);
                A[iP][h] = mul2(nPp[h], ng[h]);
                A[iM][h] = mul2(ng[h], fma2(nPp[h], r[h], nam));
                A[0][h] = mul2(naA, ng[h]);
                if constexpr (!ADJ) {
                    A[3][h] = fma2(mul2(phi[h], naA), A[0][h], A[3][h]);
                    A[4][h] = fma2(A[0][h], t, A[4][h]);
                } else {
                    A[1][h] = fma2(A[0][h], t, A[1][h]);
                    float2 kq = mul2(A[0][h], qq[h]);
                    if (PRIOR) kq = neg2(mul2(kq, na[h]));
                    const float2 f = mul2(kq, dup2(dyf));
                    A[2][h] = fma2(A[1][h], f, fma2(mul2(kq, dup2(dyvf)), kq, A[2][h]));
                    A[3][h] = add2(A[3][h], f);
                }
            }
        };

        for (int tile = 0; tile < NT; ++tile) {
            const int s = tile % NS, t0 = tile * TT;
            if (!mbar_wait(prm.wait, &full_in[s], (tile / NS) & 1, 31)) break;
            if constexpr (LOGV) {
                precisions_from_tile<T, TT, MC, CLS>(lstage(s) + warp * CLS, lam_tile + warp * CLS, prm.obs_var_min,
                                                     prm.obs_var_max, lane);
                __syncwarp();
            }
            const T *vrow = vstage(s) + cw, *lrow = lstage(s) + cw;
            const TO *dyrow = dystage(s) + cw, *dyvrow = dyvstage(s) + cw;
            const float *kqrow = kqstage(s) + j * SPT;
            if (t0 + TT <= L) {
#pragma unroll 1
                for (int t4 = 0; t4 < TT; t4 += 4) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) step(vrow, lrow, dyrow, dyvrow, kqrow, t4 + u);
                }
            } else {
                for (int tt = 0; t0 + tt < L; ++tt) step(vrow, lrow, dyrow, dyvrow, kqrow, tt);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty_in[s]);
        }

#pragma unroll
        for (int i = 0; i < SPT; ++i) {
            const int s = i * LPC + j;
            if (m < M && s < S) {
                float4 *o = reinterpret_cast<float4 *>(prm.out + (((long long)be * M + m) * S + s) * 8);
                float x[NA];
#pragma unroll
                for (int e = 0; e < NA; ++e) x[e] = pair_el(A[e], i);
                if constexpr (!ADJ) {
                    const float J = -x[3], sc = 1.0f / (1.0f + J);  // m00 + m01 = 1: folds of many records stay in range
                    o[0] = make_float4(sc, J * sc, x[2] * sc, fmaf(x[0], x[0], x[2] * J) * sc);
                    o[1] = make_float4(x[1] * sc, fmaf(x[0], x[4], x[1] * J) * sc, x[0] * sc, 0.0f);
                } else {
                    o[0] = make_float4(x[0] * x[0], x[0] * x[1], x[0], x[2]);
                    o[1] = make_float4(x[3], x[4], x[5], 0.0f);
                }
            }
        }
        // Chains that the floor of a2 binds. Here, from global memory, the walk costs the loop above no registers (inside it, or
        // as a call, up to 32), and where there are none, nothing: 33.7 us at B=2 L=1024 M=1024 float32 in 4 chunks, 34.0 without.
        if constexpr (ADJ) {
            unsigned floored = 0;
#pragma unroll
            for (int i = 0; i < SPT; ++i)
                if (m < M && pair_el(na2, i) == -kEps) floored |= 1u << i;  // (dead states have 0)
#pragma unroll 1
            for (; floored != 0; floored &= floored - 1) {
                const int s = (__ffs(floored) - 1) * LPC + j;
                walk_with_floor<T, TO, ADJ, PRIOR, LOGV>(prm, be, b, t_off, L, m, s, prm.a[(long long)m * S + s]);
            }
        }
    } else {
        // ================================================================ loader warp
        constexpr uint32_t kBytesI = sizeof(T) * TT * MC, kBytesO = sizeof(TO) * TT * MC;
        const T *vb = static_cast<const T *>(prm.v.ptr) + (long long)b * prm.v.sb + (long long)t_off * prm.v.st;
        const T *lb = static_cast<const T *>(prm.lv.ptr) + (long long)b * prm.lv.sb + (long long)t_off * prm.lv.st;
        const T *kb = static_cast<const T *>(prm.k.ptr) + (long long)b * prm.k.sb + (long long)t_off * prm.k.st;
        const T *qb = ADJ ? static_cast<const T *>(prm.q.ptr) + (long long)b * prm.q.sb + (long long)t_off * prm.q.st : nullptr;
        const TO *dyb = ADJ ? static_cast<const TO *>(prm.dy.ptr) + (long long)b * prm.dy.sb + (long long)t_off * prm.dy.st : nullptr;
        const TO *dyvb = has_dyv ? static_cast<const TO *>(prm.dyv.ptr) + (long long)b * prm.dyv.sb + (long long)t_off * prm.dyv.st : nullptr;
        if (ADJ && !has_dyv) {  // dyvar absent: its stage buffers stay zero for the whole kernel
            for (int s = 0; s < NS; ++s)
                for (int idx = lane; idx < TT * MC; idx += 32) dyvstage(s)[idx] = from_f32<TO>(0.0f);
            fence_proxy_async();
        }
        constexpr int KQP = (TT * SPAD + 31) / 32;
        float kr[KQP], qr[ADJ ? KQP : 1];
        auto load_kq = [&](int t0) {
#pragma unroll
            for (int e = 0; e < KQP; ++e) {
                const int idx = lane + e * 32, row = idx / SPAD, sidx = idx % SPAD;
                const bool in = idx < TT * SPAD && sidx < S && t0 + row < L;
                kr[e] = in ? to_f32<T>(kb[(long long)(t0 + row) * prm.k.st + sidx]) : 0.0f;
                if (ADJ) qr[e] = in ? to_f32<T>(qb[(long long)(t0 + row) * prm.q.st + sidx]) : 0.0f;
            }
        };
        int produced = 0;
        bool ok = true;
        if (NT > 0) load_kq(0);
        for (int it = 0; it < NT; ++it) {
            const int s = it % NS, t0 = it * TT;
            if (it >= NS && !mbar_wait(prm.wait, &empty_in[s], (it / NS - 1) & 1, 32, 100)) { ok = false; break; }
            if (prm.use_tma) {
                if (lane == 0) {
                    mbar_arrive_expect_tx(&full_in[s], 2 * kBytesI + (ADJ ? (has_dyv ? 2 : 1) * kBytesO : 0));
                    tma_load_3d(vstage(s), &prm.tm_v, m_cta, t_off + t0, b, &full_in[s]);
                    tma_load_3d(lstage(s), &prm.tm_lv, m_cta, t_off + t0, b, &full_in[s]);
                    if (ADJ) {
                        tma_load_3d(dystage(s), &prm.tm_dy, m_cta, t_off + t0, b, &full_in[s]);
                        if (has_dyv) tma_load_3d(dyvstage(s), &prm.tm_dyv, m_cta, t_off + t0, b, &full_in[s]);
                    }
                }
            } else {
                stage_tile<T, TT, MC, 32>(vstage(s), vb, prm.v.st, t0, L, m_cta, M, lane);
                stage_tile<T, TT, MC, 32>(lstage(s), lb, prm.lv.st, t0, L, m_cta, M, lane);
                if (ADJ) {
                    stage_tile<TO, TT, MC, 32>(dystage(s), dyb, prm.dy.st, t0, L, m_cta, M, lane);
                    if (has_dyv) stage_tile<TO, TT, MC, 32>(dyvstage(s), dyvb, prm.dyv.st, t0, L, m_cta, M, lane);
                }
            }
            float *kq = kqstage(s);
#pragma unroll
            for (int e = 0; e < KQP; ++e) {
                const int idx = lane + e * 32, row = idx / SPAD, sidx = idx % SPAD;
                if (idx < TT * SPAD) {
                    float *dst = kq + row * NK * SPAD + (sidx % LPC) * SPT + sidx / LPC;
                    dst[0] = kr[e];
                    if (ADJ) dst[SPAD] = qr[e];
                }
            }
            if (it + 1 < NT) load_kq(t0 + TT);
            if (!prm.use_tma) stage_arrive(&full_in[s]);
            if (!(prm.use_tma && lane == 0)) mbar_arrive(&full_in[s]);
            produced = it + 1;
        }
        // leaving early (a wait ran out): do not end the CTA with copies still in flight into its shared memory
        if (!ok && !prm.use_tma) cp_async_wait_all();
        if (!ok && prm.use_tma && lane == 0)
            for (int t = max(0, produced - NS); t < produced; ++t) mbar_wait(prm.wait, &full_in[t % NS], (t / NS) & 1, 33);
    }
}

}  // namespace kla
