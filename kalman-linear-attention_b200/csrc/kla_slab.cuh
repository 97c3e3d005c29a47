// Folds of per-chunk aggregates (kla_agg.cuh) for the time-parallel scan on one GPU.
#pragma once

#include "kla_common.cuh"

namespace kla {

// ---------------------------------------------------------------------------
// Folds over the chunks of one sequence held on ONE GPU (time-parallel scan).
//
// The time axis of a [B, L, ...] problem is cut into C chunks that are scanned
// as B*C independent batch entries (entry b*C + c = chunk c of batch element b),
// which fills the GPU when B*M alone does not. Each chunk needs the state it
// starts from (forward) and the carry it ends with (backward); both follow from
// the per-chunk aggregates above by a short serial fold over c, done here with
// one thread per (b, m, s) lane in float64.
//
//   forward  in:  agg [B*C, M, S, 8] (MODE 0 records), lam0/eta0 [B, M, S] or nullptr
//            out: lam_in, eta_in [B*C, M, S], the state before each chunk's first step
//   adjoint  in:  agg [B*C, M, S, 8] (MODE 1 records), dlam_fin/deta_fin [B, M, S] or nullptr, lam_in/eta_in as above
//                 or nullptr: with them the first chunk needs no record (the state it ends in is the second's start)
//            out: dlam_seed, deta_seed [B*C, M, S]: passed to the backward kernel as the gradient
//                 of each chunk's returned state, they make it start from the right carry
struct ChunkFoldParams {
    int B, C, M, S;
    const float *agg;
    const float *in_a, *in_b;
    const float *lam_in, *eta_in;  // adjoint: [B*C, M, S] start states
    float *out_a, *out_b;
};

template <bool ADJ>
__global__ void __launch_bounds__(128) kla_chunk_fold_kernel(const ChunkFoldParams prm) {
    const long long lanes = (long long)prm.M * prm.S;
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (long long)prm.B * lanes) return;
    const long long b = gid / lanes, ms = gid % lanes;
    const int C = prm.C;
    // The fold itself is serial over c, but a chunk's record does not depend on the carry: records are fetched kAhead
    // chunks before they are applied, so the loop pays C / kAhead memory latencies (16 chunks, one ahead: 7.2 us).
    constexpr int kAhead = 4;
    auto fetch = [&](int c, float4 &lo, float4 &hi) {
        const float4 *src = reinterpret_cast<const float4 *>(prm.agg + (((b * C + c) * lanes) + ms) * 8);
        lo = src[0];
        hi = src[1];
    };
    float4 lo[kAhead], hi[kAhead];  // slot i: the i-th record from here in the order of the fold
    auto fetch_nth = [&](int n, float4 &l, float4 &h) {  // record number n in that order (nothing past the last)
        l = h = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (n < (ADJ && (prm.lam_in == nullptr || C == 1) ? C : C - 1)) fetch(ADJ ? C - 1 - n : n, l, h);
    };
#pragma unroll
    for (int i = 0; i < kAhead; ++i) fetch_nth(i, lo[i], hi[i]);
    if (!ADJ) {
        // the state in homogeneous coordinates (x, w, z), P = w/x, mean = z/x: applying a record is a 3x3
        // product, and lam = x/w, eta = z/w need one reciprocal per chunk. Records are normalised, so the
        // coordinates stay far inside the float64 range for any chunk count the launcher accepts.
        double x = 1.0, w = 1.0, z = 0.0;
        if (prm.in_a != nullptr) {
            w = 1.0 / fmax((double)prm.in_a[gid], (double)kLamMin);
            z = (double)prm.in_b[gid] * w;
        }
        for (int c0 = 0; c0 < C; c0 += kAhead) {
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
                const int c = c0 + i;
                if (c >= C) break;
                const long long o = (b * C + c) * lanes + ms;
                const double rw = 1.0 / w;
                prm.out_a[o] = (float)(x * rw);
                prm.out_b[o] = (float)(z * rw);
                const float4 l = lo[i], h = hi[i];
                fetch_nth(c + kAhead, lo[i], hi[i]);
                const double nx = (double)l.x * x + (double)l.y * w, nw = (double)l.z * x + (double)l.w * w;
                z = (double)h.x * x + (double)h.y * w + (double)h.z * z;
                x = nx;
                w = nw;
            }
        }
    } else {
        const double dl = prm.in_a ? (double)prm.in_a[gid] : 0.0, de = prm.in_b ? (double)prm.in_b[gid] : 0.0;
        // (dL/dP, dL/dmean) at the end of the sequence from the gradient of (lam, eta) = (1/P, mean/P)
        const double lam = 1.0 / (double)hi[0].y, eta = (double)hi[0].z * lam;
        double cP = -lam * (lam * dl + eta * de), cm = de * lam;
        for (int n0 = 0; n0 < C; n0 += kAhead) {
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
                const int n = n0 + i;
                if (n >= C) break;
                const float4 l = lo[i], h = hi[i];
                fetch_nth(n + kAhead, lo[i], hi[i]);
                const long long o = (b * C + (C - 1 - n)) * lanes + ms;
                double P_end = h.y, mean_end = h.z;  // record: K00 K01 K11 b0 | b1 P_end mean_end
                if (n == C - 1 && n > 0 && prm.lam_in != nullptr) {
                    P_end = 1.0 / (double)prm.lam_in[o + lanes];
                    mean_end = (double)prm.eta_in[o + lanes] * P_end;
                }
                const double deta = cm * P_end;
                prm.out_b[o] = (float)deta;
                prm.out_a[o] = (float)(-(cP * P_end * P_end + mean_end * deta));
                const double nP = (double)l.x * cP + (double)l.y * cm + (double)l.w;
                cm = (double)l.z * cm + (double)h.x;
                cP = nP;
            }
        }
    }
}

}  // namespace kla
