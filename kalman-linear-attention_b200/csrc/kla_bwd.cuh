// Fused backward scan kernel: the exact adjoint of kla_fwd_kernel.
//
// Time is walked in tiles of kCkptInterval steps, last tile first. For each tile
// the forward recurrence is replayed from the tile's checkpoint, every chain's
// pre-step state (P', mean') going to shared memory, and then the adjoint is
// walked back down the tile with the two carries (dL/dP, dL/dmean) in registers.
// The forward step, in variance form (kla_common.cuh), and its derivatives
// written with the posterior (P, mean) wherever that takes fewer operations:
//
//   Pp = a2 P' + p,  g = 1/(1 + phi Pp) = P/Pp,  P = Pp g,  mean = g (a mean' + Pp r)
//   with phi = lambda_v k^2, r = lambda_v v k
//
//   mbar = c_mean + dy q                    Pbar = c_P + dyvar q^2
//   rbar = P mbar                           phibar = -P (mbar mean + Pbar P)
//   ubar = g mbar                           Ppbar = g (g Pbar + mbar w),  w = lambda_v k (v - k mean)
//   c_mean <- a ubar                        c_P <- a2 Ppbar
//   da += ubar mean'   da2 += Ppbar P'      dp += Ppbar
//   D = sum_s rbar k,  E = sum_s phibar k^2:  dv = D lambda_v,  dlambda_v = E + D v
//   dk = sum_m lambda_v (rbar v + 2 k phibar)
//
// A thread owns two neighbouring channels x SPT states. The two channels are the
// halves of every operand, so the whole walk runs on the paired fp32 instructions
// of sm_100: inputs of the step arrive as pairs, k and q are staged duplicated,
// and what a thread adds over its channels costs one addition per state. The mean
// and the P carry travel negated (n = -mean, -c_P): every product above then has
// the sign the next sum needs, since a pair instruction has no operand negation.
//
// The CTA is three groups of four warps, each with the registers its role needs
// (the register file is re-divided between the groups when the kernel starts):
//   replay warps   run the forward recurrence of tile n+1 into one of two
//                  trajectory buffers while
//   reverse warps  walk the adjoint down tile n from the other buffer, leaving
//                  what crosses threads where the trajectory was (a warp has read
//                  a step's slots before it writes them):
//                    sums over m (dk, dq): one float2 per thread and state;
//                    sums over s (D, E): one float4 per thread;
//                  sums over b and t (da, dp) stay in registers until the end;
//   helper warps   one loads (TMA tiles of v, lambda_v, dy, dy_var issued by one
//                  elected thread, and the (k, q) values of a tile, those
//                  of the next tile already in registers); three finish the sums:
//                  the CTA's channels of dk, dq and one vector atomic per (t, two
//                  states), the lane groups of dv, dlambda_v and their stores.
// Replay and reverse are different instruction streams with little in common but
// the trajectory, so running them side by side doubles the warps a scheduler can
// choose from without doubling the registers. All hand-overs go through mbarriers.
//
// With SEG a sequence is walked by several CTAs, last stretch first (SegCtl, kla_common.cuh): a CTA takes the two
// carries and the running sums for da, dp from the CTA that walked the stretch after its own, and hands its own
// on; the state its walk starts from needs no hand-over, the replay group computes it from the checkpoints.
//
// Measured on B200 at T=4096, M=1024, S=16, float32, against the kernel with one channel per thread and scalar
// arithmetic: B=8 1.42 -> 1.14 ms, B=4 0.88 -> 0.69 ms, B=16 2.59 -> 2.13 ms; 43.1 instead of 66 warp instructions per 32
// lane-steps. What bounds it is the FP32 pipe's register reads: 29 pair operations per two chains and step in the
// reverse walk and 8 in the replay, 12 and 2 of them three-operand FMAs at 3.75 cycles (kla_common.cuh), add up to about
// 230 of the 289 cycles a scheduler spends on a warp's step. Not limits: shared memory (the trajectory through tensor
// memory, a third less shared-memory traffic, takes the same 1.17 ms), the helpers (1.12 ms without their sums), the
// replay (1.08 ms without its arithmetic). Scalar FMAs in place of the pair FMAs: 1.25 ms. Fetching a step's inputs
// before the previous step's arithmetic and unrolling the whole tile gave 1.20 -> 1.17 ms; shares of dk, dq summed as halves
// and doubled once per CTA 1.148 -> 1.141.
#pragma once

#include <type_traits>

#include "kla_fwd.cuh"

namespace kla {

constexpr int kBwdStages = 3;  // input stages in flight
#ifndef KLA_REV_UNROLL
#define KLA_REV_UNROLL 8
#endif
template <int SPAD>
constexpr int kRevUnroll = SPAD > 64 ? 2 : KLA_REV_UNROLL;  // steps of the reverse walk unrolled per loop trip
#ifndef KLA_REP_UNROLL
#define KLA_REP_UNROLL 8
#endif
template <int SPAD>
constexpr int kRepUnroll = SPAD > 64 ? 2 : KLA_REP_UNROLL;  // steps of the replay unrolled per loop trip

// Registers per thread of the three warp groups after the kernel's start (BwdRegs). The kernel is compiled for
// kBwdRegsLaunch registers (384 threads, two CTAs per SM); the groups then hand registers to one another:
// 128 * (reverse + replay + helpers) must not exceed 384 * the compiled count, which the launcher checks
// against the compiled kernel before it launches (a group that asked for more than is there would wait for ever).
constexpr int kBwdRegsLaunch = 80;
#ifndef KLA_BWD_REGS_REVERSE
#define KLA_BWD_REGS_REVERSE 120
#endif
#ifndef KLA_BWD_REGS_REPLAY
#define KLA_BWD_REGS_REPLAY 72
#endif
template <int SPAD>  // at 128 states a reverse thread has twice the chains
struct BwdRegs {
    static constexpr int kReverse = SPAD > 64 ? 136 : KLA_BWD_REGS_REVERSE, kReplay = SPAD > 64 ? 64 : KLA_BWD_REGS_REPLAY;
    static constexpr int kHelper = 3 * kBwdRegsLaunch - kReverse - kReplay;
    static_assert(kHelper >= 24 && kHelper % 8 == 0 && kReverse % 8 == 0 && kReplay % 8 == 0,
                  "register counts are multiples of 8, at least 24");
    static_assert(kReplay <= kBwdRegsLaunch && kHelper <= kBwdRegsLaunch && kReverse >= kBwdRegsLaunch,
                  "two groups give registers up, one takes them");
};

template <int R>
__device__ __forceinline__ void regs_grow() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R>
__device__ __forceinline__ void regs_shrink() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}

struct alignas(64) BwdParams {
    CUtensorMap tm_v, tm_lv, tm_dy, tm_dyv;
    int B, L, M, S, NT;  // B entries; NT tiles of kCkptInterval steps = checkpoints per entry
    int use_tma;
    Tensor3 v, lv, k, q, dy, dyv, dv, dlv;
    const float *a, *p, *lam0, *eta0;
    const float2 *ckpt;
    const float *dlam_fin, *deta_fin;
    float *dk, *dq, *da, *dp, *dlam0, *deta0;
    int vec_dv, vec_dlv;
    int vec_dkq;  // two neighbouring states of dk, dq can be added to at once
    // lv holds log-variances (see FwdParams); dlv then receives the gradient with respect to them
    int lv_log_sigma;
    float obs_var_min, obs_var_max;
    WaitCtl wait;
    ChunkCtl chunk;
    SegCtl seg;  // hand: five planes [B, M, S]: the two carries and the running sums for da, da2, dp
};

// How the backward's threads cover a state size, by the number of padded states SPAD = 4 .. 128 (a power of two):
// two channels x SPT states per thread, LPC lanes per channel pair. Four states per thread only at 128, where two
// would need more than a warp per channel pair.
template <int SPAD>
struct BwdShape {
    static constexpr int kSPT = SPAD > 64 ? 4 : 2;
    static constexpr int kLPC = SPAD / kSPT;
    static constexpr int kCPW = (32 / kLPC) * 2;  // channels per warp
    static constexpr int kMC = 4 * kCPW;          // channels per CTA
    static constexpr int kCompute = 128;          // threads of a compute group
};

template <typename T, typename TO, int SPAD, int TT>
struct BwdSmem {
    using Sh = BwdShape<SPAD>;
    // bfloat16 tiles are widened once by the loader, from a ring of raw tiles into the stages: by the eight lanes and two
    // groups that read each value the conversions were a tenth of a CTA's instructions (B=8 L=4096 M=1024 S=16: 1.27 ms
    // where float32 takes 1.15). At four states the wider stages would leave room for one CTA per SM instead of two.
    static constexpr bool kWiden = sizeof(T) == 2 && SPAD >= 8;
    using TV = std::conditional_t<kWiden, float, T>;   // v, lambda_v as staged
    using TD = std::conditional_t<kWiden, float, TO>;  // dy, dyvar as staged
    static constexpr int kRawTiles = 2;
    static constexpr size_t kRawI = ((sizeof(T) * TT * Sh::kMC + 127) / 128) * 128, kRawO = ((sizeof(TO) * TT * Sh::kMC + 127) / 128) * 128;
    static constexpr size_t kRaw = kWiden ? 2 * kRawI + 2 * kRawO : 0;
    static constexpr size_t kBars = 128;
    static constexpr size_t kTileI = ((sizeof(TV) * TT * Sh::kMC + 127) / 128) * 128;  // v or lambda_v
    static constexpr size_t kTileO = ((sizeof(TD) * TT * Sh::kMC + 127) / 128) * 128;  // dy or dyvar
    static constexpr size_t kKq = sizeof(float4) * TT * SPAD;                          // (k, k, q, q) per (t, s)
    static constexpr size_t kLamF = sizeof(TV) == 4 ? 0 : ((sizeof(float) * TT * Sh::kMC + 127) / 128) * 128;  // as in FwdSmem
    static constexpr size_t kIn = 2 * kTileI + 2 * kTileO + kKq + kLamF;
    // Trajectory: a row of one float4 (P', n' of two channels) per compute thread for every (step, state). Rows are
    // padded by 64 bytes, so that helper lanes reading the same column of two neighbouring rows meet different banks.
    static constexpr int kRow = Sh::kCompute + 4;  // float4s
    static constexpr size_t kTraj = sizeof(float4) * TT * Sh::kSPT * kRow;  // one of two
    static constexpr size_t kPost = sizeof(float4) * Sh::kSPT * kRow;       // state after the last step
    static constexpr size_t kRawKq = SPAD <= 16 ? 0 : 2 * ((sizeof(T) * TT * SPAD + 127) / 128) * 128;  // k and q of a tile as they are in memory
    static constexpr size_t kTotal = kBars + kBwdStages * kIn + 2 * kTraj + kPost + 2 * kRawKq + kRawTiles * kRaw;
};

constexpr int kBwdThreads = 384;  // reverse, replay and helper groups of four warps each

// LOGV: lambda_v arrives as a log-variance (BwdParams::lv_log_sigma). A separate instantiation, so that the plain
// kernel does not carry that code.
// SEG: sequences cut into segments (BwdParams::seg, SegCtl), also a separate instantiation.
template <typename T, typename TO, int SPAD, int TT, bool PRIOR, bool LOGV, bool SEG>
__global__ void __launch_bounds__(kBwdThreads, 2) kla_bwd_kernel(const __grid_constant__ BwdParams prm) {
    using Sh = BwdShape<SPAD>;
    using Sm = BwdSmem<T, TO, SPAD, TT>;
    constexpr int SPT = Sh::kSPT, LPC = Sh::kLPC, CPW = Sh::kCPW, MC = Sh::kMC, NTC = Sh::kCompute;
    constexpr int NW = 4, NH = 4, NS = kBwdStages, ROW = Sm::kRow, CLS = 32 / LPC;
    static_assert(TT == kCkptInterval, "one checkpoint per tile");
    constexpr int kProducers = 32, kSummers = (NH - 1) * 32;
    constexpr int kStageUsers = 2 * NW + (NH - 1);  // warps that read an input stage: reverse, replay, summing helpers

    // Declared with its alignment (no run-time rounding of the pointer) so that
    // the compiler keeps every access below in the shared address space.
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *full_in = reinterpret_cast<uint64_t *>(smem);  // [NS]  loader -> everyone: stage loaded
    uint64_t *empty_in = full_in + NS;                       // [NS]  its readers -> loader: stage no longer read
    uint64_t *traj_full = empty_in + NS;                     // [2]   replay -> reverse: trajectory of a tile written
    uint64_t *part_full = traj_full + 2;                     // [2]   reverse -> summing helpers: partial sums written
    uint64_t *buf_empty = part_full + 2;                     // [2]   summing helpers -> replay: buffer reusable
    uint64_t *raw_full = buf_empty + 2;                      // [kRawTiles] bfloat16 tiles loaded, not yet widened
    static_assert((2 * NS + 6 + Sm::kRawTiles) * sizeof(uint64_t) <= Sm::kBars, "barriers fit their slot");
    using TV = typename Sm::TV;
    using TD = typename Sm::TD;
    unsigned char *in_base = smem + Sm::kBars;
    unsigned char *traj_base = in_base + NS * Sm::kIn;
    unsigned char *raw_base = traj_base + 2 * Sm::kTraj + Sm::kPost;  // two tiles of k, q as they are in memory
    float4 *post = reinterpret_cast<float4 *>(traj_base + 2 * Sm::kTraj);                                // [SPT][ROW]
    auto trajbuf = [&](int bf) { return reinterpret_cast<float4 *>(traj_base + bf * Sm::kTraj); };      // [TT*SPT][ROW]
    auto vstage = [&](int s) { return reinterpret_cast<TV *>(in_base + s * Sm::kIn); };
    auto lstage = [&](int s) { return reinterpret_cast<TV *>(in_base + s * Sm::kIn + Sm::kTileI); };
    auto dystage = [&](int s) { return reinterpret_cast<TD *>(in_base + s * Sm::kIn + 2 * Sm::kTileI); };
    auto dyvstage = [&](int s) { return reinterpret_cast<TD *>(in_base + s * Sm::kIn + 2 * Sm::kTileI + Sm::kTileO); };
    auto kqstage = [&](int s) { return reinterpret_cast<float4 *>(in_base + s * Sm::kIn + 2 * Sm::kTileI + 2 * Sm::kTileO); };
    // the precision tile the kernel computes with: float32 where lambda_v is float32 or formed from log-variances
    auto lfstage = [&](int s) {
        return reinterpret_cast<float *>(in_base + s * Sm::kIn +
                                         (sizeof(TV) == 4 ? Sm::kTileI : 2 * Sm::kTileI + 2 * Sm::kTileO + Sm::kKq));
    };
    auto lam_pair = [&](int s, int at) {
        if constexpr (sizeof(TV) == 4 || LOGV) return load_pair(lfstage(s) + at);
        else return load_pair(lstage(s) + at);
    };

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // This CTA's sequence and, when sequences are cut into segments, its stretch of it: t_off steps in, L steps long
    // (tiles and steps below count from the start of the stretch; segments are processed last-first).
    SegUnit unit{(int)blockIdx.x, (int)blockIdx.y, 0, 0};
    if constexpr (SEG) {
        unit = seg_assign(prm.seg, true);
        if (unit.seg < 0) return;
    }
    const int be = unit.b;  // batch entry: what states and checkpoints are indexed by
    const int m_cta = unit.bx * MC;
    const int M = prm.M, S = prm.S;
    const ChunkSpan span = chunk_span(prm.chunk, be, prm.L);
    const int b = span.b;
    const int t_off = SEG ? unit.seg * prm.seg.seg_len : span.t_off, tile_off = SEG ? t_off / TT : 0;
    const int L = SEG ? min(prm.seg.seg_len, prm.L - t_off) : span.L;
    const int NT = (L + TT - 1) / TT;
    const bool first_seg = !SEG || unit.seg == 0, last_seg = !SEG || unit.seg == prm.seg.nseg - 1;
    const bool has_dyv = prm.dyv.ptr != nullptr;

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(&full_in[s], Sm::kWiden ? kProducers : stage_arrivals(prm.use_tma, kProducers));
            mbar_init(&empty_in[s], kStageUsers);
        }
        for (int r = 0; r < Sm::kRawTiles; ++r) mbar_init(&raw_full[r], prm.use_tma ? 1 : stage_arrivals(false, kProducers));
        for (int bf = 0; bf < 2; ++bf) {
            mbar_init(&traj_full[bf], NW);
            mbar_init(&part_full[bf], NW);
            mbar_init(&buf_empty[bf], NH - 1);
        }
        mbar_fence_init();
    }
    __syncthreads();

    // The replay thread and the reverse thread with the same index within their groups own the same chains and the
    // same trajectory column: channels m_cta + cw, + 1 and states i * LPC + j.
    auto trow = [&](int u, int i) { return (u * SPT + i) * ROW; };

    if (warp < 2 * NW) {
        // ======================================================= the two compute groups
        const bool is_reverse = warp < NW;
        const int ctid = tid & (NTC - 1);  // index within the group
        const int cwarp = ctid >> 5;
        const int j = lane % LPC, cl = lane / LPC;
        const int cw = cwarp * CPW + cl * 2;
        const int m0 = m_cta + cw;

        // Per-chain constants as pairs over the two channels. Padding chains (s >= S or m >= M) get a = 0, p = 1.
        float2 ca[SPT], ca2[SPT], cp[SPT];
        auto load_constants = [&] {
#pragma unroll
            for (int i = 0; i < SPT; ++i) {
                const int st = i * LPC + j;
                float av[2], a2v[2], pv[2];
#pragma unroll
                for (int ci = 0; ci < 2; ++ci) {
                    const bool live = (m0 + ci < M) && (st < S);
                    av[ci] = live ? prm.a[(long long)(m0 + ci) * S + st] : 0.0f;
                    a2v[ci] = live ? fmaxf(av[ci] * av[ci], kEps) : 0.0f;
                    pv[ci] = fmaxf(live ? prm.p[(long long)(m0 + ci) * S + st] : 1.0f, kPMin);
                }
                ca[i] = make_float2(av[0], av[1]);
                ca2[i] = make_float2(a2v[0], a2v[1]);
                cp[i] = make_float2(pv[0], pv[1]);
            }
        };

        if (!is_reverse) {
            // ----------------------------------------------------------- replay
            regs_shrink<BwdRegs<SPAD>::kReplay>();
            load_constants();
            // checkpoint of the tile about to be replayed, fetched one tile ahead: (P, mean) per chain
            float2 ck[SPT][2];
            auto load_ck = [&](int tile) {
                const float2 *src = prm.ckpt + (((long long)be * prm.NT + tile_off + tile) * M + m0) * S + j;
#pragma unroll
                for (int i = 0; i < SPT; ++i)
#pragma unroll
                    for (int ci = 0; ci < 2; ++ci)
                        ck[i][ci] = (m0 + ci < M && i * LPC + j < S) ? src[ci * S + i * LPC] : make_float2(1.0f, 0.0f);
            };
            if (NT > 0) load_ck(NT - 1);

            for (int ti = 0; ti < NT; ++ti) {
                const int tile = NT - 1 - ti, s = ti % NS, bf = ti & 1;
                const int n = min(TT, L - tile * TT);
                if (!mbar_wait(prm.wait, &full_in[s], (ti / NS) & 1, 11)) break;
                if (LOGV) {  // this warp's channels of the tile: log-variance -> precision, float32
                    precisions_from_tile<TV, TT, MC, CPW>(lstage(s) + cwarp * CPW, lfstage(s) + cwarp * CPW, prm.obs_var_min,
                                                          prm.obs_var_max, lane);
                    __syncwarp();  // (in place where the stage is a bulk copy's: the loader's fence orders the two)
                }
                const TV *vrow = vstage(s) + cw;
                const float4 *kqrow = kqstage(s) + j;
                float4 *traj = trajbuf(bf) + ctid;
                float2 P[SPT], nm[SPT];
#pragma unroll
                for (int i = 0; i < SPT; ++i) {
                    P[i] = make_float2(ck[i][0].x, ck[i][1].x);
                    nm[i] = make_float2(-ck[i][0].y, -ck[i][1].y);
                }
                if (tile > 0) load_ck(tile - 1);
                // the buffer still holds the partial sums of the tile before last until the helpers have consumed them
                if (ti >= 2 && !mbar_wait(prm.wait, &buf_empty[bf], (ti / 2 - 1) & 1, 12)) break;

                auto replay_step = [&](int u) {
                    const float2 lv = lam_pair(s, u * MC + cw), nv = neg2(load_pair(vrow + u * MC));
                    float2 Pp[SPT], g[SPT], r[SPT];
#pragma unroll
                    for (int i = 0; i < SPT; ++i) {
                        const float2 k = *reinterpret_cast<const float2 *>(&kqrow[u * SPAD + i * LPC]);
                        traj[trow(u, i)] = make_float4(P[i].x, P[i].y, nm[i].x, nm[i].y);
                        float2 phi;
                        chain_inputs2(lv, nv, k, phi, r[i]);
                        g[i] = chain_denominator2(P[i], phi, ca2[i], cp[i], Pp[i]);
                    }
#pragma unroll
                    for (int i = 0; i < SPT; ++i) g[i] = rcp_approx2(g[i]);
#pragma unroll
                    for (int i = 0; i < SPT; ++i) chain_update2(P[i], nm[i], Pp[i], g[i], r[i], ca[i]);
                };
                if (n == TT) {
#pragma unroll 1
                    for (int h = 0; h < TT; h += kRepUnroll<SPAD>) {
#pragma unroll
                        for (int u = 0; u < kRepUnroll<SPAD>; ++u) replay_step(h + u);
                    }
                } else {
#pragma unroll 1
                    for (int u = 0; u < n; ++u) replay_step(u);
                }
                if (ti == 0) {  // the state after the stretch's last step: where the reverse walk starts
#pragma unroll
                    for (int i = 0; i < SPT; ++i) post[i * ROW + ctid] = make_float4(P[i].x, P[i].y, nm[i].x, nm[i].y);
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&traj_full[bf]);
                    mbar_arrive(&empty_in[s]);
                }
            }
        } else {
            // ---------------------------------------------------------- reverse
            regs_grow<BwdRegs<SPAD>::kReverse>();
            load_constants();
            // carries (that of P negated), running sums for da, da2, dp (negated), and the state after the step about
            // to be walked (P, -mean)
            float2 ncP[SPT], cm[SPT], naccA[SPT], naccA2[SPT], naccP[SPT], P[SPT], nm[SPT];
#pragma unroll
            for (int i = 0; i < SPT; ++i) {
                ncP[i] = cm[i] = naccA[i] = naccA2[i] = naccP[i] = nm[i] = make_float2(0.0f, 0.0f);
                P[i] = make_float2(1.0f, 1.0f);
            }

            for (int ti = 0; ti < NT; ++ti) {
                const int tile = NT - 1 - ti, s = ti % NS, bf = ti & 1;
                const int n = min(TT, L - tile * TT);
                if (!mbar_wait(prm.wait, &traj_full[bf], (ti / 2) & 1, 17)) break;
                if (!mbar_wait(prm.wait, &full_in[s], (ti / NS) & 1, 18)) break;
                const TV *vrow = vstage(s) + cw;
                const TD *dyrow = dystage(s) + cw;
                const TD *dyvrow = dyvstage(s) + cw;
                const float4 *kqrow = kqstage(s) + j;
                const float4 *traj = trajbuf(bf) + ctid;
                float2 *parts = reinterpret_cast<float2 *>(trajbuf(bf)) + cwarp * 64 + lane;

                if (ti == 0) {
                    // The walk starts from the state after the stretch's last step; at the end of the sequence the
                    // carries are seeded from the gradient of the returned state: lam_fin = 1/P, eta_fin = mean/P,
                    // at the end of an inner segment they and the running sums come from the segment after it.
                    bool carried = true;
                    if (!last_seg) carried = seg_wait(prm.wait, prm.seg.done + unit.seq, prm.seg.nseg - 1 - unit.seg, 19);
                    if (!carried) break;
                    const long long plane = (long long)prm.B * M * S;
#pragma unroll
                    for (int i = 0; i < SPT; ++i) {
                        const float4 fin = post[i * ROW + ctid];
                        P[i] = make_float2(fin.x, fin.y);
                        nm[i] = make_float2(fin.z, fin.w);
#pragma unroll
                        for (int ci = 0; ci < 2; ++ci) {
                            const int m = m0 + ci, st = i * LPC + j;
                            if (m >= M || st >= S) continue;
                            const long long bms = ((long long)be * M + m) * S + st;
                            auto at = [&](float2 &x) -> float & { return ci ? x.y : x.x; };
                            if (!last_seg) {
                                const float *h = prm.seg.hand + bms;
                                at(ncP[i]) = __ldcg(h);
                                at(cm[i]) = __ldcg(h + plane);
                                at(naccA[i]) = __ldcg(h + 2 * plane);
                                at(naccA2[i]) = __ldcg(h + 3 * plane);
                                at(naccP[i]) = __ldcg(h + 4 * plane);
                            } else if (prm.dlam_fin != nullptr) {
                                const float Lb = prm.dlam_fin[bms], Eb = prm.deta_fin[bms];
                                const float lam = 1.0f / at(P[i]), eta = -at(nm[i]) * lam;
                                at(cm[i]) = Eb * lam;
                                at(ncP[i]) = lam * (lam * Lb + eta * Eb);
                            }
                        }
                    }
                }

                // A step's inputs are fetched, and its gain formed, while the step before it (later in time) is in its
                // arithmetic: the stores at the end of a step could alias the next step's loads, so the compiler
                // does not move them up by itself.
                struct StepIn {
                    float2 lv, v, dy, ndyv, k[SPT], q[SPT], P[SPT], nm[SPT];  // P, nm: the state before the step
                };
                auto fetch = [&](StepIn &in, int u) {
                    in.lv = lam_pair(s, u * MC + cw);
                    in.v = load_pair(vrow + u * MC);
                    in.dy = load_pair(dyrow + u * MC);
                    in.ndyv = neg2(load_pair(dyvrow + u * MC));
#pragma unroll
                    for (int i = 0; i < SPT; ++i) {
                        const float4 kq = kqrow[u * SPAD + i * LPC];
                        in.k[i] = make_float2(kq.x, kq.y);
                        in.q[i] = make_float2(kq.z, kq.w);
                        const float4 x = traj[trow(u, i)];
                        in.P[i] = make_float2(x.x, x.y);
                        in.nm[i] = make_float2(x.z, x.w);
                    }
                };
                auto gain = [&](float2 (&g)[SPT], const StepIn &in, const float2 (&Pn)[SPT]) {  // g = P/Pp
#pragma unroll
                    for (int i = 0; i < SPT; ++i) g[i] = mul2(Pn[i], rcp_approx2(fma2(ca2[i], in.P[i], cp[i])));
                };
                // P, nm: the state after the step on entry, before it on return; nxt, gn: fetched and formed for step un
                auto reverse_step = [&](int u, const StepIn &in, const float2 (&g)[SPT], int un, StepIn &nxt, float2 (&gn)[SPT]) {
                    fetch(nxt, un);
                    const float2 nlv = neg2(in.lv), hv = mul2(in.v, dup2(0.5f)), hdy = mul2(in.dy, dup2(0.5f));
                    float2 D, E, share[SPT];
#pragma unroll
                    for (int i = 0; i < SPT; ++i) {
                        const float2 k = in.k[i], q = in.q[i];
                        const float2 e = fma2(k, nm[i], in.v);             // v - k mean
                        const float2 nw = mul2(mul2(nlv, k), e);           // -w
                        const float2 qd = mul2(q, in.ndyv);
                        float2 mbar, nPbar, dq;
                        if (PRIOR) {  // y reads a*mean and a2*P + p
                            const float2 mob = mul2(in.dy, q), nvob = mul2(qd, q);
                            mbar = fma2(mob, ca[i], cm[i]);
                            nPbar = fma2(nvob, ca2[i], ncP[i]);
                            naccA[i] = fma2(mob, nm[i], naccA[i]);
                            naccA2[i] = fma2(nvob, P[i], naccA2[i]);
                            naccP[i] = add2(naccP[i], nvob);
                            dq = fma2(qd, fma2(ca2[i], P[i], cp[i]), mul2(hdy, mul2(ca[i], nm[i])));
                        } else {
                            mbar = fma2(in.dy, q, cm[i]);
                            nPbar = fma2(qd, q, ncP[i]);
                            dq = fma2(qd, P[i], mul2(hdy, nm[i]));
                        }
                        const float2 phibar = mul2(P[i], fma2(mbar, nm[i], mul2(nPbar, P[i])));
                        const float2 rbar = mul2(P[i], mbar);
                        const float2 ubar = mul2(mbar, g[i]);
                        const float2 nPpbar = mul2(g[i], fma2(mbar, nw, mul2(nPbar, g[i])));
                        const float2 z = mul2(phibar, k);
                        const float2 dk = mul2(in.lv, fma2(rbar, hv, z));
                        D = i == 0 ? mul2(rbar, k) : fma2(rbar, k, D);
                        E = i == 0 ? mul2(z, k) : fma2(z, k, E);
                        cm[i] = mul2(ubar, ca[i]);
                        ncP[i] = mul2(nPpbar, ca2[i]);
                        naccA[i] = fma2(ubar, in.nm[i], naccA[i]);
                        naccA2[i] = fma2(nPpbar, in.P[i], naccA2[i]);
                        naccP[i] = add2(naccP[i], nPpbar);
                        P[i] = in.P[i];
                        nm[i] = in.nm[i];
                        share[i] = make_float2(dk.x + dk.y, dq.x + dq.y);  // half of this thread's dk, -dq for (t, s)
                    }
                    gain(gn, nxt, P);
                    // parked where the warp's own trajectory slots of this step were: row (u, i) of the warp is 64 float2s,
                    // the shares in its first half, D / E in the second half of rows i = 0 / 1
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < SPT; ++i) parts[2 * trow(u, i)] = share[i];
                    parts[2 * trow(u, 0) + 32] = D;
                    parts[2 * trow(u, 1) + 32] = E;
                };
                StepIn in[2];
                float2 g[2][SPT];
                fetch(in[0], n - 1);
                gain(g[0], in[0], P);
                if (n == TT) {
                    static_assert(kRevUnroll<SPAD> % 2 == 0, "the two register sets swap roles from step to step");
#pragma unroll 1
                    for (int h = TT - kRevUnroll<SPAD>; h >= 0; h -= kRevUnroll<SPAD>) {
#pragma unroll
                        for (int u = kRevUnroll<SPAD> - 1; u >= 0; --u) {
                            const int c = (kRevUnroll<SPAD> - 1 - u) & 1;
                            // (the fetch past the tile's first step re-reads that step and is not used)
                            reverse_step(h + u, in[c], g[c], max(h + u - 1, 0), in[c ^ 1], g[c ^ 1]);
                        }
                    }
                } else {
#pragma unroll 1
                    for (int u = n - 1; u >= 0; --u) {
                        reverse_step(u, in[0], g[0], max(u - 1, 0), in[1], g[1]);
                        in[0] = in[1];
#pragma unroll
                        for (int i = 0; i < SPT; ++i) g[0][i] = g[1][i];
                    }
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&part_full[bf]);
                    mbar_arrive(&empty_in[s]);
                }
            }

            if (!first_seg) {
                // ---- start of an inner segment: hand the carries and the running sums to the segment before it
                const long long plane = (long long)prm.B * M * S;
#pragma unroll
                for (int i = 0; i < SPT; ++i)
#pragma unroll
                    for (int ci = 0; ci < 2; ++ci) {
                        const int m = m0 + ci, st = i * LPC + j;
                        if (m >= M || st >= S) continue;
                        auto at = [&](const float2 &x) { return ci ? x.y : x.x; };
                        float *h = prm.seg.hand + ((long long)be * M + m) * S + st;
                        __stcg(h, at(ncP[i]));
                        __stcg(h + plane, at(cm[i]));
                        __stcg(h + 2 * plane, at(naccA[i]));
                        __stcg(h + 3 * plane, at(naccA2[i]));
                        __stcg(h + 4 * plane, at(naccP[i]));
                    }
                __threadfence();
                group_barrier_128();
                if (tid == 0) st_release_gpu(prm.seg.done + unit.seq, prm.seg.nseg - unit.seg);
            }
            // ---- start of the sequence: gradients of a, p and of the carried-in state
            if (first_seg) {
#pragma unroll
                for (int i = 0; i < SPT; ++i)
#pragma unroll
                    for (int ci = 0; ci < 2; ++ci) {
                        const int m = m0 + ci, st = i * LPC + j;
                        if (m >= M || st >= S) continue;
                        auto at = [&](const float2 &x) { return ci ? x.y : x.x; };
                        const long long ms = (long long)m * S + st, bms = ((long long)be * M + m) * S + st;
                        const float a = at(ca[i]);
                        const float da2_da = (a * a >= kEps) ? 2.0f * a : 0.0f;  // clamp_min subgradient
                        atomicAdd(prm.da + ms, -fmaf(at(naccA2[i]), da2_da, at(naccA[i])));
                        if (prm.p[ms] >= kPMin) atomicAdd(prm.dp + ms, -at(naccP[i]));
                        float lam0 = 1.0f, eta0 = 0.0f;
                        if (prm.lam0 != nullptr) {
                            lam0 = prm.lam0[bms];
                            eta0 = prm.eta0[bms];
                        }
                        // P0 = 1/max(lam0, floor), mean0 = eta0 * P0
                        const float P0 = 1.0f / fmaxf(lam0, kLamMin);
                        prm.deta0[bms] = at(cm[i]) * P0;
                        prm.dlam0[bms] = (lam0 >= kLamMin) ? (at(ncP[i]) - at(cm[i]) * eta0) * P0 * P0 : 0.0f;
                    }
            }
        }
    } else {
        // ================================================================ helpers
        regs_shrink<BwdRegs<SPAD>::kHelper>();
        const int htid = tid - 2 * NTC;
        const int hlane = htid & 31;
        constexpr uint32_t kBytesI = sizeof(T) * TT * MC, kBytesO = sizeof(TO) * TT * MC;
        int produced = 0, raw_issued = 0;
        bool ok = true;

        if (htid < kProducers) {
            // ---- loader: TMA tiles of v, lambda_v, dy, dy_var and (k, q), NS tiles ahead
            const T *vb = static_cast<const T *>(prm.v.ptr) + (long long)b * prm.v.sb + (long long)t_off * prm.v.st;
            const T *lb = static_cast<const T *>(prm.lv.ptr) + (long long)b * prm.lv.sb + (long long)t_off * prm.lv.st;
            const T *kb = static_cast<const T *>(prm.k.ptr) + (long long)b * prm.k.sb + (long long)t_off * prm.k.st;
            const T *qb = static_cast<const T *>(prm.q.ptr) + (long long)b * prm.q.sb + (long long)t_off * prm.q.st;
            const TO *dyb = static_cast<const TO *>(prm.dy.ptr) + (long long)b * prm.dy.sb + (long long)t_off * prm.dy.st;
            const TO *dyvb = has_dyv ? static_cast<const TO *>(prm.dyv.ptr) + (long long)b * prm.dyv.sb + (long long)t_off * prm.dyv.st : nullptr;
            if (!has_dyv) {  // dyvar absent: its stage buffers stay zero for the whole kernel
                for (int s = 0; s < NS; ++s)
                    for (int idx = htid; idx < TT * MC; idx += kProducers) dyvstage(s)[idx] = from_f32<TD>(0.0f);
            }
            // (k, q) of the next tile are on their way while the current one is handed over, so the loader never sits on a
            // global-memory latency: in registers up to 16 states, by per-thread asynchronous copies into shared memory
            // beyond, where a tile in registers spilled up to 500 bytes per thread, and a tile fetched when its stage was
            // free set the pace (B=4 L=2048 M=512 S=64: 1.61 and 1.10 ms, with the copies 0.80 ms). With one CTA per SM
            // the registers are the shorter way (B=4 of the headline shape 0.71 against 0.75 ms).
            constexpr int KQP = TT * SPAD / kProducers;
            constexpr bool kInRegs = KQP <= 4;
            float kr[kInRegs ? KQP : 1], qr[kInRegs ? KQP : 1];
            auto load_kq = [&](int t0) {
#pragma unroll
                for (int e = 0; e < (kInRegs ? KQP : 0); ++e) {
                    const int idx = htid + e * kProducers, row = idx / SPAD, sidx = idx % SPAD;
                    const bool in = sidx < S && t0 + row < L;
                    kr[e] = in ? to_f32<T>(kb[(long long)(t0 + row) * prm.k.st + sidx]) : 0.0f;
                    qr[e] = in ? to_f32<T>(qb[(long long)(t0 + row) * prm.q.st + sidx]) : 0.0f;
                }
            };
            auto raw = [&](int bf, int which) { return reinterpret_cast<T *>(raw_base + bf * Sm::kRawKq + which * (Sm::kRawKq / 2)); };
            auto fetch_kq = [&](int t0, int bf) {
                stage_tile<T, TT, SPAD, kProducers>(raw(bf, 0), kb, prm.k.st, t0, L, 0, S, htid);
                stage_tile<T, TT, SPAD, kProducers>(raw(bf, 1), qb, prm.q.st, t0, L, 0, S, htid);
            };
            // the four activation tiles from step t0 on into T / TO buffers; with TMA one thread arrives on `bar` with their bytes
            auto load_tiles = [&](int t0, auto *v, auto *lv, auto *dy, auto *dyv, uint64_t *bar) {
                if (prm.use_tma) {
                    if (htid == 0) {
                        if (LOGV && !Sm::kWiden) fence_proxy_async();  // the replay overwrote the log-variances in place
                        mbar_arrive_expect_tx(bar, 2 * kBytesI + (has_dyv ? 2 : 1) * kBytesO);
                        tma_load_3d(v, &prm.tm_v, m_cta, t_off + t0, b, bar);
                        tma_load_3d(lv, &prm.tm_lv, m_cta, t_off + t0, b, bar);
                        tma_load_3d(dy, &prm.tm_dy, m_cta, t_off + t0, b, bar);
                        if (has_dyv) tma_load_3d(dyv, &prm.tm_dyv, m_cta, t_off + t0, b, bar);
                    }
                } else {
                    stage_tile<T, TT, MC, kProducers>(v, vb, prm.v.st, t0, L, m_cta, M, htid);
                    stage_tile<T, TT, MC, kProducers>(lv, lb, prm.lv.st, t0, L, m_cta, M, htid);
                    stage_tile<TO, TT, MC, kProducers>(dy, dyb, prm.dy.st, t0, L, m_cta, M, htid);
                    if (has_dyv) stage_tile<TO, TT, MC, kProducers>(dyv, dyvb, prm.dyv.st, t0, L, m_cta, M, htid);
                }
            };
            // bfloat16: tile number i of the walk (v, lambda_v, dy, dy_var as which = 0 .. 3) in the raw ring, its fetch, and the
            // widening of one of its tensors
            constexpr int NR = Sm::kRawTiles;
            unsigned char *tiles_base = raw_base + 2 * Sm::kRawKq;
            auto rawtile = [&](int i, int which) {
                return reinterpret_cast<T *>(tiles_base + (i % NR) * Sm::kRaw +
                                             (which < 2 ? which * Sm::kRawI : 2 * Sm::kRawI + (which - 2) * Sm::kRawO));
            };
            auto fetch_tiles = [&](int i) {
                if constexpr (Sm::kWiden) {
                    uint64_t *bar = &raw_full[i % NR];
                    load_tiles((NT - 1 - i) * TT, rawtile(i, 0), rawtile(i, 1), reinterpret_cast<TO *>(rawtile(i, 2)),
                               reinterpret_cast<TO *>(rawtile(i, 3)), bar);
                    if (!prm.use_tma) {
                        stage_arrive(bar);
                        mbar_arrive(bar);
                    }
                    raw_issued = i + 1;
                }
            };
            auto widen = [&](const auto *src, float *dst) {
                if constexpr (sizeof(*src) == 2) {
#pragma unroll 1
                    for (int c = htid; c < TT * MC / 8; c += kProducers) {
                        const uint4 x = reinterpret_cast<const uint4 *>(src)[c];
                        const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&x);
                        const float2 f0 = __bfloat1622float2(h[0]), f1 = __bfloat1622float2(h[1]), f2 = __bfloat1622float2(h[2]),
                                     f3 = __bfloat1622float2(h[3]);
                        reinterpret_cast<float4 *>(dst)[2 * c] = make_float4(f0.x, f0.y, f1.x, f1.y);
                        reinterpret_cast<float4 *>(dst)[2 * c + 1] = make_float4(f2.x, f2.y, f3.x, f3.y);
                    }
                } else {
#pragma unroll 1
                    for (int c = htid; c < TT * MC / 4; c += kProducers) reinterpret_cast<float4 *>(dst)[c] = reinterpret_cast<const float4 *>(src)[c];
                }
            };
            if (NT > 0) {
                if (kInRegs) load_kq((NT - 1) * TT);
                else fetch_kq((NT - 1) * TT, 0);
            }
            // (widening, the walk begins NR turns early with nothing but the fetches of the first raw tiles)
#pragma unroll 1
            for (int it = Sm::kWiden ? -NR : 0; it < NT; ++it) {
                if (!Sm::kWiden || it >= 0) {
                    const int tile = NT - 1 - it, s = it % NS, t0 = tile * TT;
                    // the stage is free once the compute groups and the summing helpers are done with it
                    if (it >= NS && !mbar_wait(prm.wait, &empty_in[s], (it / NS - 1) & 1, 13, 100)) { ok = false; break; }
                    if (!kInRegs) {
                        cp_async_wait_all();  // k, q of this tile, asked for a tile ago
                        __syncwarp();
                    }
                    if constexpr (Sm::kWiden) {
                        if (!mbar_wait(prm.wait, &raw_full[it % NR], (it / NR) & 1, 16)) { ok = false; break; }
                        widen(rawtile(it, 0), vstage(s));
                        widen(rawtile(it, 1), lstage(s));
                        widen(reinterpret_cast<const TO *>(rawtile(it, 2)), dystage(s));
                        if (has_dyv) widen(reinterpret_cast<const TO *>(rawtile(it, 3)), dyvstage(s));
                    } else {
                        load_tiles(t0, vstage(s), lstage(s), dystage(s), dyvstage(s), &full_in[s]);
                        if (!prm.use_tma) stage_arrive(&full_in[s]);
                    }
                    float4 *kq = kqstage(s);
                    if (kInRegs) {
#pragma unroll
                        for (int e = 0; e < (kInRegs ? KQP : 0); ++e) kq[htid + e * kProducers] = make_float4(kr[e], kr[e], qr[e], qr[e]);
                        if (tile > 0) load_kq(t0 - TT);
                    } else {
                        if (tile > 0) fetch_kq(t0 - TT, (it + 1) & 1);
                        const T *rk = raw(it & 1, 0), *rq = raw(it & 1, 1);
#pragma unroll 8
                        for (int idx = htid; idx < TT * SPAD; idx += kProducers) {
                            const float k = to_f32<T>(rk[idx]), q = to_f32<T>(rq[idx]);
                            kq[idx] = make_float4(k, k, q, q);
                        }
                        __syncwarp();
                    }
                    // (test hook, as in the forward: the wait for tile skip_tile runs out)
                    if ((Sm::kWiden || !(prm.use_tma && htid == 0)) && !(it == prm.wait.skip_tile && htid == 1)) mbar_arrive(&full_in[s]);
                    produced = it + 1;
                }
                if constexpr (Sm::kWiden) {
                    __syncwarp();  // the raw tile has been read
                    if (it + NR < NT) fetch_tiles(it + NR);
                }
            }
        } else {
            // ---- summing helpers: finish the sums of each processed tile
            const int ctid = htid - kProducers;
            T *dvb = static_cast<T *>(prm.dv.ptr) + (long long)b * prm.dv.sb + (long long)t_off * prm.dv.st;
            T *dlvb = static_cast<T *>(prm.dlv.ptr) + (long long)b * prm.dlv.sb + (long long)t_off * prm.dlv.st;
            for (int jt = 0; jt < NT; ++jt) {
                const int tile = NT - 1 - jt, s = jt % NS, t0 = tile * TT, bf = jt & 1;
                const int n = min(TT, L - t0);
                const TV *vt = vstage(s);
                const float2 *parts = reinterpret_cast<const float2 *>(trajbuf(bf));
                if (!mbar_wait(prm.wait, &part_full[bf], (jt / 2) & 1, 14, 100)) break;
                // dk, dq: add the CTA's channels. A unit is two neighbouring states of one step (the shares of lanes
                // jj, jj + 1 of every channel pair).
                for (int unit_id = ctid; unit_id < TT * SPT * (LPC / 2); unit_id += kSummers) {
                    const int jj = (unit_id % (LPC / 2)) * 2, row = unit_id / (LPC / 2);  // row = (step, i)
                    const int u = row / SPT, st = (row % SPT) * LPC + jj;
                    const float2 *src = parts + 2 * row * ROW + jj;
                    float2 x0 = make_float2(0.0f, 0.0f), x1 = x0;
#pragma unroll
                    for (int w = 0; w < NW; ++w)
#pragma unroll
                        for (int c = 0; c < CLS; ++c) {
                            const float4 x = *reinterpret_cast<const float4 *>(src + w * 64 + c * LPC);
                            x0 = add2(x0, make_float2(x.x, x.y));
                            x1 = add2(x1, make_float2(x.z, x.w));
                        }
                    x0 = mul2(x0, make_float2(2.0f, -2.0f));  // the shares are halves of dk and -dq
                    x1 = mul2(x1, make_float2(2.0f, -2.0f));
                    if (st < S && u < n) {
                        const long long at = ((long long)b * prm.L + t_off + t0 + u) * S + st;
                        if (prm.vec_dkq) {
                            atomicAdd(reinterpret_cast<float2 *>(prm.dk + at), make_float2(x0.x, x1.x));
                            atomicAdd(reinterpret_cast<float2 *>(prm.dq + at), make_float2(x0.y, x1.y));
                        } else {
                            atomicAdd(prm.dk + at, x0.x);
                            atomicAdd(prm.dq + at, x0.y);
                            if (st + 1 < S) {
                                atomicAdd(prm.dk + at + 1, x1.x);
                                atomicAdd(prm.dq + at + 1, x1.y);
                            }
                        }
                    }
                }
                // dv, dlambda_v: add the lane group of a channel pair. v enters only through v*lambda_v
                // (kla_ops.py:177): dv = D lambda_v and dlambda_v = E + D v.
                // (threads taken from the other end, so the two loops spread over the warps)
                // A wide lane group is split over kParts threads, eight lanes each, whose sums meet by shuffles.
                constexpr int kParts = LPC > 8 ? LPC / 8 : 1, kLanes = LPC / kParts;
                static_assert(32 % kParts == 0 && (TT * (MC / 2) * kParts) % 32 == 0, "parts of a unit share a warp, whole warps work");
                for (int uidx = kSummers - 1 - ctid; uidx < TT * (MC / 2) * kParts; uidx += kSummers) {
                    const int u = uidx / (MC / 2 * kParts), pp = uidx % (MC / 2 * kParts), pr = pp / kParts, c = pr * 2;
                    const float2 *src = parts + 2 * u * SPT * ROW + (pr / CLS) * 64 + 32 + (pr % CLS) * LPC + (pp % kParts) * kLanes;
                    float2 D0 = make_float2(0.0f, 0.0f), E0 = D0;
#pragma unroll
                    for (int h = 0; h < kLanes / 2; ++h) {
                        // every other lane starts 16 bytes further on: neighbouring threads read 64 bytes (eight lanes) apart
                        const int at = 2 * ((h + (pp >> 1)) % (kLanes / 2));
                        const float4 x = *reinterpret_cast<const float4 *>(src + at);
                        const float4 y = *reinterpret_cast<const float4 *>(src + 2 * ROW + at);
                        D0 = add2(D0, add2(make_float2(x.x, x.y), make_float2(x.z, x.w)));
                        E0 = add2(E0, add2(make_float2(y.x, y.y), make_float2(y.z, y.w)));
                    }
#pragma unroll
                    for (int o = kParts / 2; o > 0; o /= 2) {
                        D0 = add2(D0, make_float2(__shfl_xor_sync(0xffffffffu, D0.x, o), __shfl_xor_sync(0xffffffffu, D0.y, o)));
                        E0 = add2(E0, make_float2(__shfl_xor_sync(0xffffffffu, E0.x, o), __shfl_xor_sync(0xffffffffu, E0.y, o)));
                    }
                    if (pp % kParts != 0 || u >= n || m_cta + c >= M) continue;
                    const float2 lam = lam_pair(s, u * MC + c), v = load_pair(vt + u * MC + c);
                    const float2 dv = mul2(D0, lam);
                    float2 dl = fma2(D0, v, E0);
                    if (LOGV) {  // chain through Lambda_v = 1 / min(softplus(x) + floor, ceiling)
                        dl.x *= precision_slope(lam.x, prm.obs_var_min, prm.obs_var_max);
                        dl.y *= precision_slope(lam.y, prm.obs_var_min, prm.obs_var_max);
                    }
                    T *p0 = dvb + (long long)(t0 + u) * prm.dv.st + m_cta + c;
                    T *p1 = dlvb + (long long)(t0 + u) * prm.dlv.st + m_cta + c;
                    const bool full = m_cta + c + 1 < M;
                    if (full && prm.vec_dv) {
                        store_pair(p0, dv.x, dv.y);
                    } else {
                        p0[0] = from_f32<T>(dv.x);
                        if (full) p0[1] = from_f32<T>(dv.y);
                    }
                    if (full && prm.vec_dlv) {
                        store_pair(p1, dl.x, dl.y);
                    } else {
                        p1[0] = from_f32<T>(dl.x);
                        if (full) p1[1] = from_f32<T>(dl.y);
                    }
                }
                __syncwarp();
                if (hlane == 0) {
                    mbar_arrive(&buf_empty[bf]);
                    mbar_arrive(&empty_in[s]);
                }
            }
        }
        if (!ok) cp_async_wait_all();
        if (!ok && prm.use_tma && htid == 0) {
            if (Sm::kWiden)
                for (int t = max(0, raw_issued - Sm::kRawTiles); t < raw_issued; ++t)
                    mbar_wait(prm.wait, &raw_full[t % Sm::kRawTiles], (t / Sm::kRawTiles) & 1, 15);
            else
                for (int t = max(0, produced - NS); t < produced; ++t) mbar_wait(prm.wait, &full_in[t % NS], (t / NS) & 1, 15);
        }
    }
}

}  // namespace kla
