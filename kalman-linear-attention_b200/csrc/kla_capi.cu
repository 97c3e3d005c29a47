// extern "C" entry points of libkla_b200.so: argument checks, kernel-shape
// selection and launches. No torch types, no allocation, no exceptions.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "../../include/kla_b200.h"
#include "kla_block.cuh"
#include "kla_conv_bwd.cuh"
#include "kla_decode.cuh"
#include "kla_epilogue.cuh"
#include "kla_launch.cuh"
#include "kla_linear.cuh"
#include "kla_rawscan.cuh"
#include "kla_slab.cuh"
#include "kla_step.cuh"
#include "kla_token.cuh"

// The device's status word (kla_b200_device_status). Kernels get its device address in their
// parameters (WaitCtl::status): in host code the name below is only a handle.
static __device__ int g_kla_status = 0;

namespace {

using namespace kla;

std::atomic<long long> g_launches{0};
thread_local cudaError_t g_last_cuda = cudaSuccess;
thread_local char g_errbuf[256];
// KLA_B200_NO_TMA=1 forces the plain-load staging path (used by the tests to cover it)
const bool g_no_tma = [] { const char *e = getenv("KLA_B200_NO_TMA"); return e && e[0] == '1'; }();

int cuda_fail(cudaError_t e) {
    g_last_cuda = e;
    return KLA_B200_ECUDA;
}

// A launch that may start before the kernel in front of it has ended (programmatic dependent launch): the kernel itself
// waits (grid_dep_wait) before it touches anything that kernel could have written.
template <typename Params>
cudaError_t launch_dependent(void (*kern)(const Params), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, const Params &prm) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, prm);
}

Tensor3 t3(const kla_b200_tensor3 &t) { return Tensor3{t.ptr, t.stride_b, t.stride_t}; }

bool aligned(const void *p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// Vector stores of 2 output elements are legal when every row start is aligned to them.
template <typename T>
int vec2_ok(const kla_b200_tensor3 &t) {
    return t.ptr != nullptr && aligned(t.ptr, 2 * sizeof(T)) && (t.stride_b % 2) == 0 && (t.stride_t % 2) == 0;
}

// cuTensorMapEncodeTiled is fetched from the driver at run time, so the library
// links against the CUDA runtime only.
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// Rank-3 tensor map over a [B, L, M] activation tensor, dims (M, L, B), box
// (box_m, box_t, 1). Returns false when the tensor does not meet the TMA rules
// (16-byte aligned base and strides); the kernels then stage with plain loads.
template <typename T>
bool make_tile_map(CUtensorMap *tm, const kla_b200_tensor3 &t, int64_t B, int64_t L, int64_t M, int box_m, int box_t) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (enc == nullptr || t.ptr == nullptr || B <= 0 || L <= 0 || M <= 0) return false;
    // size-1 dimensions may carry arbitrary strides; give them the dense value
    const int64_t st = L > 1 ? t.stride_t : M;
    const int64_t sb = B > 1 ? t.stride_b : L * st;
    const uint64_t st_b = (uint64_t)st * sizeof(T), sb_b = (uint64_t)sb * sizeof(T);
    if (!aligned(t.ptr, 16) || st_b % 16 || sb_b % 16 || st < M || st_b >= (1ull << 40) || sb_b >= (1ull << 40))
        return false;
    if ((box_m * sizeof(T)) % 16 || box_m > 256 || box_t > 256) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)M, (cuuint64_t)L, (cuuint64_t)B};
    const cuuint64_t strides[2] = {st_b, sb_b};
    const cuuint32_t box[3] = {(cuuint32_t)box_m, (cuuint32_t)box_t, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUtensorMapDataType dt = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    return enc(tm, dt, 3, t.ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int lpc_for(int64_t S) {
    int lpc = 1;
    while ((int64_t)kSPT * lpc < S) lpc *= 2;
    return lpc;  // 1..32 for S <= 128
}

bool known_type(int32_t dtype) { return dtype == KLA_B200_F32 || dtype == KLA_B200_BF16; }

int check_common(int64_t B, int64_t L, int64_t M, int64_t S, int32_t in_dtype, int32_t out_dtype) {
    if (B < 0 || L < 0 || M < 0 || S < 0) return KLA_B200_EINVAL;
    if (S > KLA_B200_MAX_DSTATE) return KLA_B200_EUNSUPPORTED;
    if (!known_type(in_dtype) || !known_type(out_dtype)) return KLA_B200_EUNSUPPORTED;
    if (in_dtype == KLA_B200_F32 && out_dtype == KLA_B200_BF16) return KLA_B200_EUNSUPPORTED;
    if (B > 65535 || L > (1 << 30) || M > (1 << 30)) return KLA_B200_EUNSUPPORTED;
    return KLA_B200_OK;
}

// rows of t can be read and written two elements at a time
bool pair_ok(const kla_b200_tensor3 &t, size_t esz) {
    return (reinterpret_cast<uintptr_t>(t.ptr) % (2 * esz)) == 0 && t.stride_b % 2 == 0 && t.stride_t % 2 == 0;
}

// A sequence of L steps cut into `chunks` pieces of chunk_len steps (the last one may be shorter); chunks <= 1: whole.
int check_chunks(int64_t B, int64_t L, int64_t chunks, int64_t chunk_len, ChunkCtl *cc) {
    *cc = ChunkCtl{1, (int)L};
    if (chunks <= 1) return chunks < 0 ? KLA_B200_EINVAL : KLA_B200_OK;
    if (chunk_len <= 0 || chunk_len > L || chunks > L || (chunks - 1) * chunk_len >= L || chunks * chunk_len < L) return KLA_B200_EINVAL;
    if (B * chunks > 65535) return KLA_B200_EUNSUPPORTED;
    *cc = ChunkCtl{(int)chunks, (int)chunk_len};
    return KLA_B200_OK;
}

// One launch that clears up to five stretches of words, in place of as many memory-set operations.
constexpr int kZeroRanges = 5;
struct ZeroParams {
    int *ptr[kZeroRanges];
    unsigned long long end[kZeroRanges];  // running totals of the stretches' words
};
__global__ void __launch_bounds__(256) kla_zero_kernel(const __grid_constant__ ZeroParams prm) {
    const unsigned long long n = prm.end[kZeroRanges - 1];
    for (unsigned long long i = (unsigned long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (unsigned long long)gridDim.x * 256) {
        unsigned long long from = 0;
#pragma unroll
        for (int r = 0; r < kZeroRanges; ++r) {
            if (i >= from && i < prm.end[r]) prm.ptr[r][i - from] = 0;
            from = prm.end[r];
        }
    }
}
struct ZeroList {
    ZeroParams prm{};
    int n = 0;
    void add(void *p, size_t words) {
        if (words == 0) return;
        prm.ptr[n] = static_cast<int *>(p);
        prm.end[n] = (n ? prm.end[n - 1] : 0) + words;
        ++n;
    }
    cudaError_t run(cudaStream_t st) {
        if (n == 0) return cudaSuccess;
        for (int r = n; r < kZeroRanges; ++r) { prm.end[r] = prm.end[n - 1]; prm.ptr[r] = prm.ptr[0]; }
        const unsigned long long blocks = (prm.end[kZeroRanges - 1] + 1023) / 1024;
        kla_zero_kernel<<<(unsigned)(blocks < 1184 ? blocks : 1184), 256, 0, st>>>(prm);
        return cudaGetLastError();
    }
};

int check_t3(const kla_b200_tensor3 &t, size_t esz, bool required) {
    if (t.ptr == nullptr) return required ? KLA_B200_EINVAL : KLA_B200_OK;
    if (!aligned(t.ptr, esz)) return KLA_B200_EALIGN;
    if (t.stride_b < 0 || t.stride_t < 0) return KLA_B200_EINVAL;
    return KLA_B200_OK;
}

constexpr int kMaxDevices = 64;
std::mutex g_symbol_mu;
int *g_status_ptr[kMaxDevices] = {};
// test hooks (kla_b200_test_hooks): wait limit and the tile whose hand-over the loader leaves incomplete
std::atomic<unsigned> g_wait_limit_ns{1000000000u};
std::atomic<int> g_skip_tile{-1};

// Device address of the status word on the current device (looked up on first use), with the current
// wait settings. Returns a C-ABI status.
int wait_ctl(WaitCtl *w) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e);
    if (dev < 0 || dev >= kMaxDevices) return KLA_B200_EUNSUPPORTED;
    {
        std::lock_guard<std::mutex> lock(g_symbol_mu);
        if (g_status_ptr[dev] == nullptr) {
            void *ptr = nullptr;
            e = cudaGetSymbolAddress(&ptr, g_kla_status);
            if (e != cudaSuccess) return cuda_fail(e);
            g_status_ptr[dev] = static_cast<int *>(ptr);
        }
        w->status = g_status_ptr[dev];
    }
    w->limit_ns = g_wait_limit_ns.load();
    w->skip_tile = g_skip_tile.load();
    return KLA_B200_OK;
}

// ---- sequences cut into segments (SegCtl, kla_common.cuh): the scratch behind the checkpoints and the plan
//   [forward: ticket (256 B) | done, one int per (b, m)] [backward: the same] [forward hand-over: float2 per lane]
//   [backward hand-over: 5 floats per lane]
constexpr size_t kSegAlign = 256;
size_t seg_round(size_t n) { return (n + kSegAlign - 1) / kSegAlign * kSegAlign; }
struct SegScratch {
    size_t flags;   // bytes of one direction's ticket + done block
    size_t hand_f;  // offset of the forward's hand-over records
    size_t hand_b;  // offset of the backward's
    size_t total;
};
// false when the sizes do not fit size_t
bool seg_scratch(int64_t B, int64_t M, int64_t S, SegScratch *out) {
    if (B <= 0 || M <= 0 || S <= 0) { *out = SegScratch{0, 0, 0, 0}; return true; }
    const size_t bm = (size_t)B * (size_t)M;  // B <= 65535 and M <= 2^30 (check_common)
    if (bm > SIZE_MAX / ((size_t)S * 64)) return false;
    const size_t lanes = bm * (size_t)S;
    out->flags = kSegAlign + seg_round(bm * sizeof(int));
    out->hand_f = 2 * out->flags;
    out->hand_b = out->hand_f + seg_round(lanes * sizeof(float2));
    out->total = out->hand_b + seg_round(lanes * 5 * sizeof(float));
    return true;
}
size_t ckpt_part_bytes(int64_t B, int64_t L, int64_t M, int64_t S) {
    const int64_t nt = (L + kCkptInterval - 1) / kCkptInterval;
    // saturating product: a size that does not fit size_t reads as SIZE_MAX, never as a small number
    size_t n = sizeof(float2);
    for (const int64_t f : {B, nt, M, S}) {
        if (n > SIZE_MAX / (size_t)f) return SIZE_MAX;
        n *= (size_t)f;
    }
    return n > SIZE_MAX - kSegAlign ? SIZE_MAX : seg_round(n);
}

// How many segments for `ctas` sequences of L steps (and their length). Segments pay when the sequences do not
// fill the SMs' CTA slots evenly. Measured on B200 at T=4096, M=1024, S=16 (ms without -> with): backward, two
// CTAs per SM: B=8 1.50 -> 1.42, B=10 2.35 -> 1.68, B=12 2.35 -> 1.96, B=14 2.97 -> 2.32, B=16 2.96 -> 2.60;
// forward, four per SM: B=10 0.62 -> 0.59, B=14 0.81 -> 0.65, B=16 0.81 -> 0.71, but B=8 0.44 -> 0.55: with
// fewer sequences than half its slots the waiting CTAs spread the running ones unevenly over the SMs. So: the
// backward whenever there are more sequences than SMs (16 segments up to two per SM, else 8), the forward from
// two sequences per SM on. KLA_B200_SEGMENTS=0 switches segments off, =N asks for N in both kernels.
// forced: -1 = the policy above, 0 / 1 = off, N = N segments. sms: SMs of the device.
int plan_segments_for(int64_t ctas, int64_t L, bool backward, int sms, int forced, int *seg_len) {
    *seg_len = (int)L;
    if (forced == 0 || forced == 1 || L <= 0) return 1;
    int want = 8;
    int64_t min_len = 256;  // shorter segments cost more in hand-overs than they even out (chunks of 256 steps: no gain)
    if (forced > 1) {
        want = forced;
        min_len = kTT;
    } else {
        if (sms <= 0 || ctas <= (backward ? sms : 2 * sms)) return 1;
        if (backward && ctas <= 2 * sms) want = 16;
    }
    int64_t len = (L + want - 1) / want;
    len = (len + kTT - 1) / kTT * kTT;  // whole tiles of both kernels (and whole checkpoint intervals)
    if (len < min_len) len = min_len;
    const int64_t n = (L + len - 1) / len;
    if (n < 2 || n > 65535) return 1;
    *seg_len = (int)len;
    return (int)n;
}

int plan_segments(int64_t ctas, int64_t L, bool backward, int *seg_len) {
    const char *env = getenv("KLA_B200_SEGMENTS");  // read per launch: the tests switch it within one process
    const int forced = env != nullptr ? atoi(env) : -1;
    return plan_segments_for(ctas, L, backward, forced < 0 ? device_sms() : 0, forced, seg_len);
}

// Fill prm.seg for one direction; its ticket and done words go on the list of what to clear before the launch. The working memory is the bytes behind the
// checkpoints, or, for a forward without checkpoints, the caller's `work` buffer of the same layout.
template <typename Params>
int seg_setup(Params &prm, void *ckpt, void *work, int64_t B, int64_t L, int64_t M, int64_t S, int mc, bool backward,
              ZeroList &zero) {
    prm.seg = SegCtl{1, (int)L, nullptr, nullptr, nullptr};
    if ((ckpt == nullptr && work == nullptr) || L <= 0 || prm.chunk.n > 1) return KLA_B200_OK;
    const int64_t ctas = ((M + mc - 1) / mc) * B;
    int seg_len = (int)L;
    const int nseg = plan_segments(ctas, L, backward, &seg_len);
    if (nseg <= 1) return KLA_B200_OK;
    SegScratch sc;
    if (!seg_scratch(B, M, S, &sc)) return KLA_B200_OK;
    const size_t base = ckpt != nullptr ? ckpt_part_bytes(B, L, M, S) : 0;
    if (base == SIZE_MAX) return KLA_B200_OK;
    unsigned char *p = static_cast<unsigned char *>(ckpt != nullptr ? ckpt : work) + base;
    unsigned char *flags = p + (backward ? sc.flags : 0);
    zero.add(flags, sc.flags / sizeof(int));
    prm.seg.nseg = nseg;
    prm.seg.seg_len = seg_len;
    prm.seg.ticket = reinterpret_cast<int *>(flags);
    prm.seg.done = reinterpret_cast<int *>(flags + kSegAlign);
    prm.seg.hand = reinterpret_cast<float *>(p + (backward ? sc.hand_b : sc.hand_f));
    return KLA_B200_OK;
}

// Tensor maps of the forward's tiles (box: the CTA's channels x one tile of steps), then the launch.
template <typename T, typename TO, int LPC, bool PRIOR>
int prep_fwd(FwdParams &prm, const kla_b200_fwd_args &a, cudaStream_t st) {
    const int mc = scan_channels_per_cta(LPC);
    ZeroList zero;
    if (int rc = seg_setup(prm, a.ckpt, a.work, a.B, a.L, a.M, a.S, mc, false, zero)) return rc;
    if (const cudaError_t e = zero.run(st); e != cudaSuccess) return cuda_fail(e);
    prm.use_tma = !g_no_tma && make_tile_map<T>(&prm.tm_v, a.v, a.B, a.L, a.M, mc, kTT) &&
                  make_tile_map<T>(&prm.tm_lv, a.lambda_v, a.B, a.L, a.M, mc, kTT);
    if (prm.epilogue)  // z and gate tiles travel like v and lambda_v when they meet the tensor-map rules
        prm.epi_tma = !g_no_tma && (a.z.ptr == nullptr || make_tile_map<T>(&prm.tm_z, a.z, a.B, a.L, a.M, mc, kTT)) &&
                      (a.gate.ptr == nullptr || make_tile_map<T>(&prm.tm_gate, a.gate, a.B, a.L, a.M, mc, kTT));
    const cudaError_t e = launch_fwd<T, TO, LPC, PRIOR>(prm, st);
    g_launches++;
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

template <typename T, typename TO, int LPC, bool PRIOR>
int prep_bwd(BwdParams &prm, const kla_b200_bwd_args &a, cudaStream_t st) {
    const int mc = bwd_channels_per_cta<LPC>();
    ZeroList zero;
    zero.add(a.dk, (size_t)a.B * a.L * a.S);
    zero.add(a.dq, (size_t)a.B * a.L * a.S);
    zero.add(a.da, (size_t)a.M * a.S);
    zero.add(a.dp, (size_t)a.M * a.S);
    if (int rc = seg_setup(prm, const_cast<void *>(a.ckpt), nullptr, a.B, a.L, a.M, a.S, mc, true, zero)) return rc;
    if (const cudaError_t e = zero.run(st); e != cudaSuccess) return cuda_fail(e);
    prm.use_tma = !g_no_tma && make_tile_map<T>(&prm.tm_v, a.v, a.B, a.L, a.M, mc, kBwdTT) &&
                  make_tile_map<T>(&prm.tm_lv, a.lambda_v, a.B, a.L, a.M, mc, kBwdTT) &&
                  make_tile_map<TO>(&prm.tm_dy, a.dy, a.B, a.L, a.M, mc, kBwdTT) &&
                  (a.dy_var.ptr == nullptr || make_tile_map<TO>(&prm.tm_dyv, a.dy_var, a.B, a.L, a.M, mc, kBwdTT));
    const cudaError_t e = launch_bwd<T, TO, LPC, PRIOR>(prm, st);
    g_launches++;
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

template <typename T, typename TO, int LPC, bool PRIOR>
int launch_step(const StepParams &prm, cudaStream_t st) {
    const long long threads = (long long)prm.B * prm.M * LPC;
    if ((threads + 127) / 128 > 0x7fffffffll) return KLA_B200_EUNSUPPORTED;  // grid.x limit
    const unsigned blocks = (unsigned)((threads + 127) / 128);
    kla_step_kernel<T, TO, LPC, PRIOR><<<blocks, 128, 0, st>>>(prm);
    g_launches++;
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

// Expand (dtype pair, lanes per channel, prior flag) into a template instantiation.
#define KLA_DISPATCH_LPC(FN, T, TO, PRIOR, lpc, ...)          \
    switch (lpc) {                                            \
        case 1: return FN<T, TO, 1, PRIOR>(__VA_ARGS__);      \
        case 2: return FN<T, TO, 2, PRIOR>(__VA_ARGS__);      \
        case 4: return FN<T, TO, 4, PRIOR>(__VA_ARGS__);      \
        case 8: return FN<T, TO, 8, PRIOR>(__VA_ARGS__);      \
        case 16: return FN<T, TO, 16, PRIOR>(__VA_ARGS__);    \
        case 32: return FN<T, TO, 32, PRIOR>(__VA_ARGS__);    \
        default: return KLA_B200_EUNSUPPORTED;                \
    }
#define KLA_DISPATCH_PRIOR(FN, T, TO, prior, lpc, ...)                  \
    if (prior) { KLA_DISPATCH_LPC(FN, T, TO, true, lpc, __VA_ARGS__) }  \
    else { KLA_DISPATCH_LPC(FN, T, TO, false, lpc, __VA_ARGS__) }
#define KLA_DISPATCH(FN, din, dout, prior, lpc, ...)                                         \
    do {                                                                                     \
        if ((din) == KLA_B200_F32 && (dout) == KLA_B200_F32) {                               \
            KLA_DISPATCH_PRIOR(FN, float, float, prior, lpc, __VA_ARGS__)                    \
        } else if ((din) == KLA_B200_BF16 && (dout) == KLA_B200_F32) {                       \
            KLA_DISPATCH_PRIOR(FN, __nv_bfloat16, float, prior, lpc, __VA_ARGS__)            \
        } else if ((din) == KLA_B200_BF16 && (dout) == KLA_B200_BF16) {                      \
            KLA_DISPATCH_PRIOR(FN, __nv_bfloat16, __nv_bfloat16, prior, lpc, __VA_ARGS__)    \
        } else {                                                                             \
            return KLA_B200_EUNSUPPORTED;                                                    \
        }                                                                                    \
    } while (0)

int dispatch_fwd(int din, int dout, bool prior, int lpc, FwdParams &prm, const kla_b200_fwd_args &a, cudaStream_t st) {
    KLA_DISPATCH(prep_fwd, din, dout, prior, lpc, prm, a, st);
}
int dispatch_bwd(int din, int dout, bool prior, int lpc, BwdParams &prm, const kla_b200_bwd_args &a, cudaStream_t st) {
    KLA_DISPATCH(prep_bwd, din, dout, prior, lpc, prm, a, st);
}
// Tensor maps of the aggregate kernel's tiles, then the launch.
template <typename T, typename TO, int LPC, bool PRIOR>
int prep_agg(AggParams &prm, const kla_b200_slab_args &a, cudaStream_t st) {
    const int mc = agg_channels_per_cta(LPC);
    const bool adj = a.adjoint != 0;
    prm.use_tma = !g_no_tma && a.L > 0 && make_tile_map<T>(&prm.tm_v, a.v, a.B, a.L, a.M, mc, kAggTT) &&
                  make_tile_map<T>(&prm.tm_lv, a.lambda_v, a.B, a.L, a.M, mc, kAggTT) &&
                  (!adj || (make_tile_map<TO>(&prm.tm_dy, a.dy, a.B, a.L, a.M, mc, kAggTT) &&
                            (a.dy_var.ptr == nullptr || make_tile_map<TO>(&prm.tm_dyv, a.dy_var, a.B, a.L, a.M, mc, kAggTT))));
    const cudaError_t e = launch_agg<T, TO, LPC, PRIOR>(prm, adj, st);
    g_launches++;
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}
int dispatch_slab(int din, int dout, bool prior, int lpc, AggParams &prm, const kla_b200_slab_args &a, cudaStream_t st) {
    KLA_DISPATCH(prep_agg, din, dout, prior, lpc, prm, a, st);
}
int dispatch_step(int din, int dout, bool prior, int lpc, const StepParams &prm, cudaStream_t st) {
    KLA_DISPATCH(launch_step, din, dout, prior, lpc, prm, st);
}
template <typename T, typename TO, int LPC, bool PRIOR>
int launch_step_layer(const StepLayerParams &prm, cudaStream_t st) {
    auto go = [&](auto kern, int channels) -> int {
        const long long blocks = (long long)prm.B * ((prm.M + channels - 1) / channels);
        if (blocks > 0x7fffffffll) return KLA_B200_EUNSUPPORTED;  // grid.x limit
        const cudaError_t e = launch_dependent(kern, dim3((unsigned)blocks), 128, 0, st, prm);
        g_launches++;
        return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
    };
    // Four channels per thread once that still leaves every SM two CTAs; below, the CTAs' latency is the time.
    if ((long long)prm.B * prm.M >= 2ll * device_sms() * kStepLayerChannels<LPC, 4>)
        return go(kla_step_layer_kernel<T, TO, LPC, PRIOR, 4>, kStepLayerChannels<LPC, 4>);
    return go(kla_step_layer_kernel<T, TO, LPC, PRIOR, 1>, kStepLayerChannels<LPC, 1>);
}
int dispatch_step_layer(int din, int dout, bool prior, int lpc, const StepLayerParams &prm, cudaStream_t st) {
    KLA_DISPATCH(launch_step_layer, din, dout, prior, lpc, prm, st);
}

}  // namespace

namespace {
template <class Op, bool WIDE>
int launch_rawscan_as(const kla_b200_rawscan_args *a, void *stream);

template <class Op>
int launch_rawscan(const kla_b200_rawscan_args *a, void *stream, bool takes_state0, bool gives_dstate0) {
    if (a == nullptr || a->B < 0 || a->L < 0 || a->N < 0) return KLA_B200_EINVAL;
    if (a->B > 65535 || a->L > (1 << 30) || a->N > (1 << 30)) return KLA_B200_EUNSUPPORTED;
    if ((!takes_state0 && a->state0 != nullptr) || (!gives_dstate0 && a->dstate0 != nullptr)) return KLA_B200_EINVAL;
    for (int i = 0; i < Op::NIN; ++i) {
        if (a->in[i] == nullptr) return KLA_B200_EINVAL;
        if (!aligned(a->in[i], sizeof(float))) return KLA_B200_EALIGN;
    }
    for (int k = 0; k < Op::NOUT; ++k) {
        if (a->out[k] == nullptr) return KLA_B200_EINVAL;
        if (!aligned(a->out[k], sizeof(float))) return KLA_B200_EALIGN;
    }
    if (a->B == 0 || a->N == 0) return KLA_B200_OK;
    if (Op::NIN >= 6 && (a->N + kRawLC - 1) / kRawLC * a->B <= device_sms()) return launch_rawscan_as<Op, false>(a, stream);
    return launch_rawscan_as<Op, true>(a, stream);
}

template <class Op, bool WIDE>
int launch_rawscan_as(const kla_b200_rawscan_args *a, void *stream) {
    constexpr int kRawTT = RawTile<Op, WIDE>::TT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    RawParams prm{};
    prm.B = (int)a->B; prm.L = (int)a->L; prm.N = (int)a->N;
    prm.NT = (int)((a->L + kRawTT - 1) / kRawTT);
    prm.state0 = a->state0; prm.dstate0 = a->dstate0;
    bool tma = !g_no_tma && a->L > 0;
    for (int i = 0; i < Op::NIN; ++i) {
        prm.in[i] = a->in[i];
        const kla_b200_tensor3 t{const_cast<float *>(a->in[i]), a->L * a->N, a->N};
        tma = tma && make_tile_map<float>(&prm.tm_in[i], t, a->B, a->L, a->N, kRawLC, kRawTT + (i == Op::HALO ? 1 : 0));
    }
    for (int k = 0; k < Op::NOUT; ++k) {
        prm.out[k] = a->out[k];
        const kla_b200_tensor3 t{a->out[k], a->L * a->N, a->N};
        tma = tma && make_tile_map<float>(&prm.tm_out[k], t, a->B, a->L, a->N, kRawLC, kRawTT);
    }
    prm.use_tma = tma;
    if (int rc = wait_ctl(&prm.wait)) return rc;
    prm.wait.skip_tile = -1;  // the hook is for the fused scan kernels
    auto kern = kla_rawscan_kernel<Op, WIDE>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RawSmem<Op, WIDE>::kTotal);
    if (e != cudaSuccess) return cuda_fail(e);
    dim3 grid((unsigned)((a->N + kRawLC - 1) / kRawLC), (unsigned)a->B);
    kern<<<grid, kRawLC + 32, RawSmem<Op, WIDE>::kTotal, st>>>(prm);
    g_launches++;
    e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

template <int NT, int RT, int MODE, bool NORM>
int launch_linear(const LinearParams &prm, cudaStream_t st) {
    auto kern = kla_linear_kernel<NT, RT, MODE, NORM>;
    const size_t smem = kLinearRedBytes<NT, RT> + linear_x_bytes(kLinearStaged<NT, NORM>, NT, prm.K);
    if (smem > KLA_B200_LINEAR_SMEM) return KLA_B200_EUNSUPPORTED;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, KLA_B200_LINEAR_SMEM);
        if (e != cudaSuccess) return cuda_fail(e);
    }
    const int n_out = MODE == kLinearSwiglu ? prm.N / 2 : prm.N;
    // A CTA per tile up to two per SM, which is what fits; beyond, a CTA walks several tiles, the next one's W on its way
    // while it adds up the last one.
    constexpr int rows = MODE == kLinearSwiglu ? 16 : 16 * RT;
    const int tiles = (n_out + rows - 1) / rows, most = 2 * device_sms();
    const cudaError_t e = launch_dependent(kern, dim3((unsigned)(tiles < most ? tiles : most)), kLinearWarps * 32, smem, st, prm);
    g_launches++;
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}
// Tiles of W per CTA: one while x is small beside them or the tiles would not fill the SMs, else two, since every CTA
// brings in all of x.
template <int NT, int MODE, bool NORM>
int dispatch_linear_tiles(const LinearParams &prm, cudaStream_t st) {
    if constexpr (MODE == kLinearSwiglu) return launch_linear<NT, 2, MODE, NORM>(prm, st);
    else if constexpr (NT < 4) return launch_linear<NT, 1, MODE, NORM>(prm, st);
    else return prm.N > 16 * device_sms() ? launch_linear<NT, 2, MODE, NORM>(prm, st) : launch_linear<NT, 1, MODE, NORM>(prm, st);
}
template <int NT>
int dispatch_linear(const LinearParams &prm, int mode, cudaStream_t st) {
    const bool norm = prm.norm_w != nullptr;
    if (mode == kLinearSwiglu) return norm ? dispatch_linear_tiles<NT, kLinearSwiglu, true>(prm, st) : dispatch_linear_tiles<NT, kLinearSwiglu, false>(prm, st);
    if (mode == kLinearConv) return norm ? dispatch_linear_tiles<NT, kLinearConv, true>(prm, st) : dispatch_linear_tiles<NT, kLinearConv, false>(prm, st);
    return norm ? dispatch_linear_tiles<NT, kLinearPlain, true>(prm, st) : dispatch_linear_tiles<NT, kLinearPlain, false>(prm, st);
}

// Where the words between the phases of a token lie in its working memory.
struct TokenWork {
    size_t proj, sens, y, xa, xb, h, total;
};
TokenWork token_work(const kla_b200_token_args *a) {
    int64_t proj = 0, sens = 0, y = 0, h = 0;
    for (int64_t i = 0; i < a->layers; ++i) {
        const kla_b200_token_layer &l = a->layer[i];
        const int64_t p = (l.gated ? 2 : 1) * l.M, s = l.w_value + l.M + 2 * l.S;
        proj = p > proj ? p : proj;
        sens = s > sens ? s : sens;
        y = l.M > y ? l.M : y;
        h = l.hidden > h ? l.hidden : h;
    }
    TokenWork w{};
    size_t at = kTokHeader;
    auto place = [&](int64_t columns) {
        const size_t here = at;
        at += ((size_t)a->B * columns * sizeof(uint32_t) + 255) / 256 * 256;
        return here;
    };
    w.proj = place(proj); w.sens = place(sens); w.y = place(y); w.xa = place(a->d); w.xb = place(a->d); w.h = place(a->mlp ? h : 0);
    w.total = at;
    return w;
}

int64_t token_widest(const kla_b200_token_args *a) {  // columns of the widest projection, whose x has to fit shared memory
    int64_t K = a->d;
    for (int64_t i = 0; i < a->layers; ++i) {
        K = a->layer[i].M > K ? a->layer[i].M : K;
        if (a->mlp && a->layer[i].hidden > K) K = a->layer[i].hidden;
    }
    return K;
}

int check_token(const kla_b200_token_args *a) {
    if (a == nullptr || a->B < 0 || a->d < 0 || a->layers < 0 || (a->layers > 0 && !a->layer)) return KLA_B200_EINVAL;
    if (a->B > KLA_B200_TOKEN_MAX_ROWS || a->layers > KLA_B200_TOKEN_MAX_LAYERS || a->d % 8 || a->d > (1 << 20)) return KLA_B200_EUNSUPPORTED;
    for (int64_t i = 0; i < a->layers; ++i) {
        const kla_b200_token_layer &l = a->layer[i];
        if (l.M < 0 || l.S < 0 || l.hidden < 0 || l.w_value < 0 || l.lambda_skip_len < 0) return KLA_B200_EINVAL;
        if (l.M % 8 || l.M > (1 << 18) || l.S > KLA_B200_MAX_DSTATE || (a->mlp && (l.hidden % 8 || l.hidden > (1 << 18)))) return KLA_B200_EUNSUPPORTED;
        if (l.M == 0 || l.S == 0 || (l.w_value != 0 && l.w_value != l.M) || (a->mlp && (l.hidden == 0 || !l.norm_weight))) return KLA_B200_EINVAL;
        if (l.conv_weight && (l.conv_taps < 1 || l.conv_taps > KLA_B200_MAX_CONV_TAPS)) return KLA_B200_EUNSUPPORTED;
        if (l.conv_activation < KLA_B200_ACT_SILU || l.conv_activation > KLA_B200_ACT_NONE || l.gate_activation < KLA_B200_ACT_SILU ||
            l.gate_activation > KLA_B200_ACT_NONE)
            return KLA_B200_EINVAL;
        if (l.lambda_skip_len != 0 && l.lambda_skip_len != 1 && l.lambda_skip_len != l.M) return KLA_B200_EINVAL;
    }
    const int widest = (int)token_widest(a);
    return token_ring(widest) ? KLA_B200_OK : KLA_B200_EUNSUPPORTED;
}

template <int LAYERS>
int launch_token(const kla_b200_token_args *a, cudaStream_t st) {
    using bf16 = __nv_bfloat16;
    TokenParams<LAYERS> prm{};
    const int B = (int)a->B, d = (int)a->d, G = device_sms();
    const bool mlp = a->mlp != 0;
    const TokenWork w = token_work(a);
    auto words = [&](size_t offset) { return reinterpret_cast<uint32_t *>(static_cast<char *>(a->work) + offset); };
    uint32_t *xa = words(w.xa), *xb = words(w.xb), *h = words(w.h);
    prm.B = B; prm.layers = (int)a->layers; prm.phases = mlp ? 5 : 3; prm.norm_eps = a->norm_eps;
    prm.out_var = static_cast<bf16 *>(a->y_var);
    prm.proj = words(w.proj); prm.sens = words(w.sens); prm.y = words(w.y); prm.sync = words(0);
    if (int rc = wait_ctl(&prm.wait)) return rc;
    for (int i = 0; i < prm.layers; ++i) {
        const kla_b200_token_layer &l = a->layer[i];
        TokenLayer &t = prm.layer[i];
        const int M = (int)l.M, S = (int)l.S, hidden = (int)l.hidden, N_in = (l.gated ? 2 : 1) * M, N_sensor = l.w_value + M + 2 * S;
        const bool first = i == 0, last = i + 1 == prm.layers;
        auto phase = [&](int k, const void *weight, const void *bias, const void *norm, int N, int K, const void *src, int64_t src_sb, void *dst, int dst_sb) {
            TokenPhase &p = t.ph[k];
            p.w = static_cast<const bf16 *>(weight); p.bias = static_cast<const bf16 *>(bias); p.norm_w = static_cast<const bf16 *>(norm);
            p.src = src; p.src_sb = src_sb; p.dst = dst; p.dst_sb = dst_sb; p.N = N; p.K = K;
            const int octs = (N + 7) / 8;
            p.oct_q = octs / G; p.oct_r = octs % G;
        };
        // x: what the layer starts from, words of the layer before (their last projection's outputs)
        const void *x = first ? a->x : mlp ? xb : xa;
        const int64_t x_sb = first ? a->x_stride_b : d;
        void *mixed = last && !mlp ? a->out : xa, *sum = last ? a->out : xb;
        phase(kTokIn, l.in_weight, l.in_bias, l.norm_weight, N_in, d, x, x_sb, prm.proj, N_in);
        phase(kTokSensor, l.sensor_weight, l.sensor_bias, nullptr, N_sensor, M, prm.proj, N_in, prm.sens, N_sensor);
        phase(kTokOut, l.out_weight, l.out_bias, nullptr, d, M, prm.y, M, mixed, d);
        t.ph[kTokIn].plain_src = first;
        t.ph[kTokOut].plain_dst = last && !mlp;
        if (l.norm_weight) { t.ph[kTokOut].res = x; t.ph[kTokOut].res_sb = x_sb; t.ph[kTokOut].plain_res = first; }
        if (mlp) {
            phase(kTokGateUp, l.w12, l.b12, l.mlp_norm_weight, hidden, d, xa, d, h, hidden);
            phase(kTokDown, l.w3, l.b3, nullptr, d, hidden, h, hidden, sum, d);
            t.ph[kTokDown].res = xa; t.ph[kTokDown].res_sb = d; t.ph[kTokDown].plain_dst = last;
        }
        t.conv_w = l.conv_weight; t.conv_b = l.conv_bias; t.conv_state = static_cast<bf16 *>(l.conv_state);
        t.a = l.a; t.p = l.p; t.skip = l.lambda_skip_len ? l.lambda_skip : nullptr; t.lam = l.lam; t.eta = l.eta;
        t.M = M; t.S = S; t.taps = (int)l.conv_taps; t.conv_act = l.conv_activation;
        t.gate_act = l.gate_activation; t.gated = l.gated != 0; t.skip_len = l.lambda_skip_len; t.w_value = l.w_value;
        t.qk_norm = l.qk_norm; t.prior = l.decode_from_prior;
        t.vec = S % 4 == 0 && aligned(l.a, 16) && aligned(l.p, 16) && aligned(l.lam, 16) && aligned(l.eta, 16);
        t.lpc = 1;
        while (4 * t.lpc < S) t.lpc *= 2;
        const int channels = 32 / t.lpc;
        t.blocks = (M + channels - 1) / channels;
        t.unit_q = B * t.blocks / (G * kTokWarps); t.unit_r = B * t.blocks % (G * kTokWarps);
        t.obs_var_min = l.obs_var_min; t.obs_var_max = l.obs_var_max; t.clip = l.clip_value;
    }
    prm.ring = token_ring((int)token_widest(a));
    const size_t smem = token_smem((int)token_widest(a), prm.ring);
    auto kern = kla_token_kernel<LAYERS>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e);
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;  // CTAs wait for one another's words
    attr.val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)G);
    cfg.blockDim = dim3(kTokThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, prm);
    g_launches++;
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}
}  // namespace


extern "C" {

int64_t kla_b200_ckpt_interval(void) { return kCkptInterval; }

size_t kla_b200_ckpt_bytes(int64_t B, int64_t L, int64_t M, int64_t S) {
    if (B <= 0 || L <= 0 || M <= 0 || S <= 0) return 0;
    if (B > 65535 || M > (1 << 30)) return SIZE_MAX;
    const size_t ck = ckpt_part_bytes(B, L, M, S);
    SegScratch sc;
    if (ck == SIZE_MAX || !seg_scratch(B, M, S, &sc) || ck > SIZE_MAX - sc.total) return SIZE_MAX;
    return ck + sc.total;
}

int kla_b200_plan_segments(int64_t sequences, int64_t L, int backward, int sms, int forced, int *seg_len) {
    int len = 0;
    const int n = plan_segments_for(sequences, L, backward != 0, sms, forced, &len);
    if (seg_len != nullptr) *seg_len = len;
    return n;
}

size_t kla_b200_segment_scratch_bytes(int64_t B, int64_t M, int64_t S) {
    SegScratch sc;
    if (B > 65535 || M > (1 << 30) || !seg_scratch(B, M, S, &sc)) return SIZE_MAX;
    return sc.total;
}

int kla_b200_scan_fwd(const kla_b200_fwd_args *a, void *stream) {
    if (a == nullptr) return KLA_B200_EINVAL;
    int rc = check_common(a->B, a->L, a->M, a->S, a->in_dtype, a->out_dtype);
    if (rc) return rc;
    const size_t esz = a->in_dtype == KLA_B200_F32 ? 4 : 2, osz = a->out_dtype == KLA_B200_F32 ? 4 : 2;
    const bool empty = a->B == 0 || a->M == 0 || a->S == 0;
    if (empty) return KLA_B200_OK;
    if (!a->a || !a->p || !a->lam_fin || !a->eta_fin) return KLA_B200_EINVAL;
    if ((a->lam0 == nullptr) != (a->eta0 == nullptr)) return KLA_B200_EINVAL;
    if (a->L > 0) {
        const kla_b200_tensor3 *ts[] = {&a->v, &a->lambda_v, &a->k, &a->q};
        for (const kla_b200_tensor3 *t : ts)
            if ((rc = check_t3(*t, esz, true))) return rc;
        if ((rc = check_t3(a->y, osz, true))) return rc;
        if ((rc = check_t3(a->y_var, osz, true))) return rc;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    FwdParams prm{};
    if ((rc = check_chunks(a->B, a->L, a->chunks, a->chunk_len, &prm.chunk))) return rc;
    prm.B = (int)a->B * prm.chunk.n; prm.L = (int)a->L; prm.M = (int)a->M; prm.S = (int)a->S;
    prm.NC = (int)((prm.chunk.len + kCkptInterval - 1) / kCkptInterval);
    prm.v = t3(a->v); prm.lv = t3(a->lambda_v); prm.k = t3(a->k); prm.q = t3(a->q);
    prm.y = t3(a->y); prm.yv = t3(a->y_var);
    prm.a = a->a; prm.p = a->p; prm.lam0 = a->lam0; prm.eta0 = a->eta0;
    prm.lam_fin = a->lam_fin; prm.eta_fin = a->eta_fin;
    prm.sequence_state = prm.chunk.n > 1 && a->sequence_state != 0;
    prm.ckpt = static_cast<float2 *>(a->ckpt);
    prm.lv_log_sigma = a->lambda_v_is_log_variance != 0;
    prm.obs_var_min = a->obs_var_min; prm.obs_var_max = a->obs_var_max;
    {
        const bool has_skip = a->lambda_skip_len != 0, has_gate = a->gate.ptr != nullptr;
        if (has_skip || has_gate) {
            // with a backward to follow, the scan's own outputs must be kept for the epilogue's adjoint
            // (the gate's adjoint reads them; the skip path alone does not)
            if (a->ckpt != nullptr && has_gate && (a->y_raw.ptr == nullptr || a->y_var_raw.ptr == nullptr)) return KLA_B200_EUNSUPPORTED;
            if ((a->y_raw.ptr == nullptr) != (a->y_var_raw.ptr == nullptr)) return KLA_B200_EINVAL;
            if (a->y_raw.ptr != nullptr) {
                if ((rc = check_t3(a->y_raw, osz, true)) || (rc = check_t3(a->y_var_raw, osz, true))) return rc;
                prm.y_raw = t3(a->y_raw); prm.yv_raw = t3(a->y_var_raw);
                prm.vec_raw = osz == 4 ? vec2_ok<float>(a->y_raw) && vec2_ok<float>(a->y_var_raw)
                                       : vec2_ok<__nv_bfloat16>(a->y_raw) && vec2_ok<__nv_bfloat16>(a->y_var_raw);
            }
            if (has_skip && ((a->lambda_skip_len != 1 && a->lambda_skip_len != a->M) || !a->lambda_skip || !a->z.ptr))
                return KLA_B200_EINVAL;
            if (a->gate_activation < KLA_B200_ACT_SILU || a->gate_activation > KLA_B200_ACT_NONE) return KLA_B200_EINVAL;
            if (has_skip && (rc = check_t3(a->z, esz, true))) return rc;
            if (has_gate && (rc = check_t3(a->gate, esz, true))) return rc;
            prm.epilogue = 1;
            if (has_skip) { prm.z = t3(a->z); prm.skip = a->lambda_skip; prm.skip_len = a->lambda_skip_len; }
            if (has_gate) { prm.gate = t3(a->gate); prm.gate_act = a->gate_activation; }
        }
    }
    if ((rc = wait_ctl(&prm.wait))) return rc;
    prm.vec_y = a->out_dtype == KLA_B200_F32 ? vec2_ok<float>(a->y) : vec2_ok<__nv_bfloat16>(a->y);
    prm.vec_yv = a->out_dtype == KLA_B200_F32 ? vec2_ok<float>(a->y_var) : vec2_ok<__nv_bfloat16>(a->y_var);
    return dispatch_fwd(a->in_dtype, a->out_dtype, a->decode_from_prior != 0, lpc_for(a->S), prm, *a, st);
}

int kla_b200_scan_bwd(const kla_b200_bwd_args *a, void *stream) {
    if (a == nullptr) return KLA_B200_EINVAL;
    int rc = check_common(a->B, a->L, a->M, a->S, a->in_dtype, a->out_dtype);
    if (rc) return rc;
    const size_t esz = a->in_dtype == KLA_B200_F32 ? 4 : 2, osz = a->out_dtype == KLA_B200_F32 ? 4 : 2;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t n_bls = (size_t)a->B * a->L * a->S, n_ms = (size_t)a->M * a->S, n_bms = (size_t)a->B * a->M * a->S;
    if (n_bls && (!a->dk || !a->dq)) return KLA_B200_EINVAL;
    if (n_ms && (!a->da || !a->dp)) return KLA_B200_EINVAL;
    if (n_bms && (!a->dlam0 || !a->deta0)) return KLA_B200_EINVAL;
    if ((a->lam0 == nullptr) != (a->eta0 == nullptr)) return KLA_B200_EINVAL;
    if ((a->dlam_fin == nullptr) != (a->deta_fin == nullptr)) return KLA_B200_EINVAL;
    cudaError_t e;
    if (n_bms == 0 || a->L == 0) {  // no kernel below: the sums are empty
        ZeroList zero;
        zero.add(a->dk, n_bls);
        zero.add(a->dq, n_bls);
        zero.add(a->da, n_ms);
        zero.add(a->dp, n_ms);
        if ((e = zero.run(st)) != cudaSuccess) return cuda_fail(e);
    }
    if (n_bms == 0) return KLA_B200_OK;
    if (a->L == 0) {  // nothing to scan: the state gradient passes straight through
        if (a->dlam_fin) {
            if ((e = cudaMemcpyAsync(a->dlam0, a->dlam_fin, n_bms * 4, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return cuda_fail(e);
            if ((e = cudaMemcpyAsync(a->deta0, a->deta_fin, n_bms * 4, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return cuda_fail(e);
        } else {
            if ((e = cudaMemsetAsync(a->dlam0, 0, n_bms * 4, st)) != cudaSuccess) return cuda_fail(e);
            if ((e = cudaMemsetAsync(a->deta0, 0, n_bms * 4, st)) != cudaSuccess) return cuda_fail(e);
        }
        return KLA_B200_OK;
    }
    if (!a->a || !a->p || !a->ckpt) return KLA_B200_EINVAL;
    const kla_b200_tensor3 *ts[] = {&a->v, &a->lambda_v, &a->k, &a->q, &a->dv, &a->dlambda_v};
    for (const kla_b200_tensor3 *t : ts)
        if ((rc = check_t3(*t, esz, true))) return rc;
    if ((rc = check_t3(a->dy, osz, true))) return rc;
    if ((rc = check_t3(a->dy_var, osz, false))) return rc;

    BwdParams prm{};
    if ((rc = check_chunks(a->B, a->L, a->chunks, a->chunk_len, &prm.chunk))) return rc;
    prm.B = (int)a->B * prm.chunk.n; prm.L = (int)a->L; prm.M = (int)a->M; prm.S = (int)a->S;
    prm.NT = (int)((prm.chunk.len + kBwdTT - 1) / kBwdTT);
    prm.v = t3(a->v); prm.lv = t3(a->lambda_v); prm.k = t3(a->k); prm.q = t3(a->q);
    prm.dy = t3(a->dy); prm.dyv = t3(a->dy_var); prm.dv = t3(a->dv); prm.dlv = t3(a->dlambda_v);
    prm.a = a->a; prm.p = a->p; prm.lam0 = a->lam0; prm.eta0 = a->eta0;
    prm.ckpt = static_cast<const float2 *>(a->ckpt);
    prm.lv_log_sigma = a->lambda_v_is_log_variance != 0;
    prm.obs_var_min = a->obs_var_min; prm.obs_var_max = a->obs_var_max;
    prm.dlam_fin = a->dlam_fin; prm.deta_fin = a->deta_fin;
    prm.dk = a->dk; prm.dq = a->dq; prm.da = a->da; prm.dp = a->dp;
    prm.dlam0 = a->dlam0; prm.deta0 = a->deta0;
    if ((rc = wait_ctl(&prm.wait))) return rc;
    prm.vec_dv = a->in_dtype == KLA_B200_F32 ? vec2_ok<float>(a->dv) : vec2_ok<__nv_bfloat16>(a->dv);
    prm.vec_dkq = a->S % 2 == 0 && aligned(a->dk, 8) && aligned(a->dq, 8);
    prm.vec_dlv = a->in_dtype == KLA_B200_F32 ? vec2_ok<float>(a->dlambda_v) : vec2_ok<__nv_bfloat16>(a->dlambda_v);
    return dispatch_bwd(a->in_dtype, a->out_dtype, a->decode_from_prior != 0, lpc_for(a->S), prm, *a, st);
}

int kla_b200_slab_aggregate(const kla_b200_slab_args *a, void *stream) {
    if (a == nullptr) return KLA_B200_EINVAL;
    int rc = check_common(a->B, a->L, a->M, a->S, a->in_dtype, a->out_dtype);
    if (rc) return rc;
    if (a->B == 0 || a->M == 0 || a->S == 0) return KLA_B200_OK;
    if (!a->a || !a->p || !a->out) return KLA_B200_EINVAL;
    if ((a->lam0 == nullptr) != (a->eta0 == nullptr)) return KLA_B200_EINVAL;
    const size_t esz = a->in_dtype == KLA_B200_F32 ? 4 : 2, osz = a->out_dtype == KLA_B200_F32 ? 4 : 2;
    if (a->L > 0) {
        if ((rc = check_t3(a->v, esz, true)) || (rc = check_t3(a->lambda_v, esz, true)) || (rc = check_t3(a->k, esz, true)))
            return rc;
        if (a->adjoint && ((rc = check_t3(a->q, esz, true)) || (rc = check_t3(a->dy, osz, true)) ||
                           (rc = check_t3(a->dy_var, osz, false))))
            return rc;
    }
    AggParams prm{};
    if ((rc = check_chunks(a->B, a->L, a->chunks, a->chunk_len, &prm.chunk))) return rc;
    prm.B = (int)a->B * prm.chunk.n; prm.L = (int)a->L; prm.M = (int)a->M; prm.S = (int)a->S;
    prm.v = t3(a->v); prm.lv = t3(a->lambda_v); prm.k = t3(a->k); prm.q = t3(a->q);
    prm.dy = t3(a->dy); prm.dyv = t3(a->dy_var);
    prm.a = a->a; prm.p = a->p; prm.lam0 = a->lam0; prm.eta0 = a->eta0; prm.out = a->out;
    prm.lv_log_sigma = a->lambda_v_is_log_variance != 0;
    prm.obs_var_min = a->obs_var_min; prm.obs_var_max = a->obs_var_max;
    if ((rc = wait_ctl(&prm.wait))) return rc;
    prm.wait.skip_tile = -1;  // the hook is for the scan kernels
    return dispatch_slab(a->in_dtype, a->out_dtype, a->decode_from_prior != 0, lpc_for(a->S), prm, *a,
                         static_cast<cudaStream_t>(stream));
}

int kla_b200_epilogue_bwd(const kla_b200_epilogue_bwd_args *a, void *stream) {
    if (a == nullptr || a->B < 0 || a->L < 0 || a->M < 0) return KLA_B200_EINVAL;
    if (a->in_dtype != KLA_B200_F32 && a->in_dtype != KLA_B200_BF16) return KLA_B200_EUNSUPPORTED;
    if (a->out_dtype != KLA_B200_F32 && a->out_dtype != KLA_B200_BF16) return KLA_B200_EUNSUPPORTED;
    if (a->in_dtype == KLA_B200_F32 && a->out_dtype == KLA_B200_BF16) return KLA_B200_EUNSUPPORTED;
    if (a->B > 65535 || a->L > (1 << 30) || a->M > (1 << 30)) return KLA_B200_EUNSUPPORTED;
    if (a->gate_activation < KLA_B200_ACT_SILU || a->gate_activation > KLA_B200_ACT_NONE) return KLA_B200_EINVAL;
    const bool has_skip = a->lambda_skip_len != 0, has_gate = a->gate.ptr != nullptr;
    if (has_skip && ((a->lambda_skip_len != 1 && a->lambda_skip_len != a->M) || !a->lambda_skip || !a->dlambda_skip)) return KLA_B200_EINVAL;
    const size_t esz = a->in_dtype == KLA_B200_F32 ? 4 : 2, osz = a->out_dtype == KLA_B200_F32 ? 4 : 2;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e;
    const bool empty = a->B == 0 || a->L == 0 || a->M == 0, wide_sum = a->lambda_skip_len == 1 && a->work != nullptr && !empty;
    if (wide_sum && !aligned(a->work, 8)) return KLA_B200_EALIGN;
    if (has_skip && (e = wide_sum ? cudaMemsetAsync(a->work, 0, sizeof(SkipSum), st)
                                  : cudaMemsetAsync(a->dlambda_skip, 0, sizeof(float) * (size_t)a->lambda_skip_len, st)) != cudaSuccess)
        return cuda_fail(e);
    if (empty) return KLA_B200_OK;
    int rc;
    if ((rc = check_t3(a->dout, osz, true)) || (rc = check_t3(a->dout_var, osz, false)) || (rc = check_t3(a->dy, osz, true)) ||
        (rc = check_t3(a->dy_var, osz, true)))
        return rc;
    if (has_gate && ((rc = check_t3(a->gate, esz, true)) || (rc = check_t3(a->dgate, esz, true)) ||
                     (rc = check_t3(a->y_raw, osz, true)) || (rc = check_t3(a->y_var_raw, osz, true))))
        return rc;
    if (has_skip && ((rc = check_t3(a->z, esz, true)) || (rc = check_t3(a->dz, esz, true)))) return rc;
    const long long row_blocks = (a->L + kEpiRows - 1) / kEpiRows;
    if (row_blocks > 65535) return KLA_B200_EUNSUPPORTED;
    EpilogueBwdParams prm{};
    prm.B = (int)a->B; prm.L = (int)a->L; prm.M = (int)a->M;
    prm.dout = t3(a->dout); prm.dout_var = t3(a->dout_var); prm.y_raw = t3(a->y_raw); prm.yv_raw = t3(a->y_var_raw);
    if (has_skip) { prm.z = t3(a->z); prm.dz = t3(a->dz); prm.skip = a->lambda_skip; prm.skip_len = a->lambda_skip_len; prm.dskip = a->dlambda_skip; }
    static_assert(sizeof(SkipSum) == KLA_B200_SKIP_SUM_BYTES, "as the header says");
    prm.sum = wide_sum ? static_cast<SkipSum *>(a->work) : nullptr;
    if (has_gate) { prm.gate = t3(a->gate); prm.dgate = t3(a->dgate); prm.gate_act = a->gate_activation; }
    prm.dy = t3(a->dy); prm.dy_var = t3(a->dy_var);
    // four channels per thread when every tensor can be read and written as 4-element vectors, eight when they are all
    // bfloat16 and 8-element ones
    auto vec_ok = [&](const kla_b200_tensor3 &t, size_t sz, int n) {
        return t.ptr == nullptr || (aligned(t.ptr, n * sz) && t.stride_b % n == 0 && t.stride_t % n == 0);
    };
    auto all_ok = [&](int n) {
        return a->M % n == 0 && vec_ok(a->dout, osz, n) && vec_ok(a->dout_var, osz, n) && vec_ok(a->dy, osz, n) &&
               vec_ok(a->dy_var, osz, n) && (!has_gate || (vec_ok(a->gate, esz, n) && vec_ok(a->dgate, esz, n) &&
               vec_ok(a->y_raw, osz, n) && vec_ok(a->y_var_raw, osz, n))) && (!has_skip || (vec_ok(a->z, esz, n) && vec_ok(a->dz, esz, n)));
    };
    const int per = osz == 2 && all_ok(8) ? 8 : all_ok(4) ? 4 : 1;
    // few rows per CTA until many of them would still give every SM four CTAs
    const int64_t columns = (a->M + 128 * per - 1) / (128 * per);
    const bool few = columns * a->B * row_blocks < 4 * device_sms();
    const int rows = few ? kEpiFewRows : kEpiRows;
    dim3 grid((unsigned)columns, (unsigned)((a->L + rows - 1) / rows), (unsigned)a->B);
#define KLA_EPI_ROWS(T, TO, VEC, Z, G)                                                                   \
    do {                                                                                                 \
        if (few) kla_epilogue_bwd_kernel<T, TO, VEC, kEpiFewRows, Z, G><<<grid, 128, 0, st>>>(prm);       \
        else kla_epilogue_bwd_kernel<T, TO, VEC, kEpiRows, Z, G><<<grid, 128, 0, st>>>(prm);              \
    } while (0)
#define KLA_EPI_HALVES(T, TO, VEC)                                \
    do {                                                          \
        if (has_skip && has_gate) KLA_EPI_ROWS(T, TO, VEC, true, true); \
        else if (has_skip) KLA_EPI_ROWS(T, TO, VEC, true, false); \
        else KLA_EPI_ROWS(T, TO, VEC, false, true);               \
    } while (0)
#define KLA_EPI_LAUNCH(T, TO)                   \
    do {                                        \
        if (per == 4) KLA_EPI_HALVES(T, TO, 4); \
        else KLA_EPI_HALVES(T, TO, 1);          \
    } while (0)
    if (!has_skip && !has_gate) return KLA_B200_EINVAL;  // nothing to differentiate
    if (a->in_dtype == KLA_B200_F32) KLA_EPI_LAUNCH(float, float);
    else if (a->out_dtype == KLA_B200_F32) KLA_EPI_LAUNCH(__nv_bfloat16, float);
    else if (per == 8) KLA_EPI_HALVES(__nv_bfloat16, __nv_bfloat16, 8);
    else KLA_EPI_LAUNCH(__nv_bfloat16, __nv_bfloat16);
#undef KLA_EPI_HALVES
#undef KLA_EPI_ROWS
#undef KLA_EPI_LAUNCH
    g_launches++;
    e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

int kla_b200_chunk_fold(const kla_b200_chunk_fold_args *a, void *stream) {
    if (a == nullptr || a->B < 0 || a->C < 1 || a->M < 0 || a->S < 0) return KLA_B200_EINVAL;
    if (a->S > KLA_B200_MAX_DSTATE || a->B * a->C > 65535 || a->M > (1 << 30)) return KLA_B200_EUNSUPPORTED;
    if (a->B == 0 || a->M == 0 || a->S == 0) return KLA_B200_OK;
    if (!a->agg || !a->out_a || !a->out_b || (a->in_a == nullptr) != (a->in_b == nullptr) || (a->lam_in == nullptr) != (a->eta_in == nullptr))
        return KLA_B200_EINVAL;
    if (!aligned(a->agg, 16)) return KLA_B200_EALIGN;
    ChunkFoldParams prm{};
    prm.B = (int)a->B; prm.C = (int)a->C; prm.M = (int)a->M; prm.S = (int)a->S;
    prm.agg = a->agg; prm.in_a = a->in_a; prm.in_b = a->in_b; prm.lam_in = a->lam_in; prm.eta_in = a->eta_in; prm.out_a = a->out_a; prm.out_b = a->out_b;
    const long long lanes = a->B * a->M * a->S;
    const unsigned blocks = (unsigned)((lanes + 127) / 128);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (a->adjoint) kla_chunk_fold_kernel<true><<<blocks, 128, 0, st>>>(prm);
    else kla_chunk_fold_kernel<false><<<blocks, 128, 0, st>>>(prm);
    g_launches++;
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

int kla_b200_step(const kla_b200_step_args *a, void *stream) {
    if (a == nullptr) return KLA_B200_EINVAL;
    int rc = check_common(a->B, 1, a->M, a->S, a->in_dtype, a->out_dtype);
    if (rc) return rc;
    if (a->B == 0 || a->M == 0) return KLA_B200_OK;
    if (!a->v || !a->lambda_v || !a->y || !a->y_var || !a->a || !a->p) return KLA_B200_EINVAL;
    if (a->S > 0 && (!a->k || !a->q || !a->lam || !a->eta || !a->lam_out || !a->eta_out)) return KLA_B200_EINVAL;
    const size_t esz = a->in_dtype == KLA_B200_F32 ? 4 : 2, osz = a->out_dtype == KLA_B200_F32 ? 4 : 2;
    const void *ps[] = {a->v, a->lambda_v, a->k, a->q};
    for (const void *p : ps)
        if (p && !aligned(p, esz)) return KLA_B200_EALIGN;
    if (!aligned(a->y, osz) || !aligned(a->y_var, osz)) return KLA_B200_EALIGN;
    StepParams prm{};
    prm.B = (int)a->B; prm.M = (int)a->M; prm.S = (int)a->S;
    prm.v = a->v; prm.lv = a->lambda_v; prm.k = a->k; prm.q = a->q;
    prm.v_sb = a->v_stride_b; prm.lv_sb = a->lambda_v_stride_b; prm.k_sb = a->k_stride_b; prm.q_sb = a->q_stride_b;
    prm.a = a->a; prm.p = a->p; prm.lam = a->lam; prm.eta = a->eta;
    prm.y = a->y; prm.yv = a->y_var; prm.lam_out = a->lam_out; prm.eta_out = a->eta_out;
    prm.vec = a->S % 4 == 0 && aligned(a->lam, 16) && aligned(a->eta, 16) && aligned(a->a, 16) && aligned(a->p, 16) &&
              aligned(a->lam_out, 16) && aligned(a->eta_out, 16);
    int lpc = 1;
    while (lpc * 4 < a->S) lpc *= 2;
    return dispatch_step(a->in_dtype, a->out_dtype, a->decode_from_prior != 0, lpc, prm, static_cast<cudaStream_t>(stream));
}

int kla_b200_conv_step(const kla_b200_conv_step_args *a, void *stream) {
    if (a == nullptr || a->B < 0 || a->D < 0) return KLA_B200_EINVAL;
    if (a->K < 1 || a->K > KLA_B200_MAX_CONV_TAPS) return KLA_B200_EUNSUPPORTED;
    if (a->dtype != KLA_B200_F32 && a->dtype != KLA_B200_BF16) return KLA_B200_EUNSUPPORTED;
    if (a->activation < KLA_B200_ACT_SILU || a->activation > KLA_B200_ACT_NONE) return KLA_B200_EINVAL;
    if (a->B == 0 || a->D == 0) return KLA_B200_OK;
    if (!a->x || !a->weight || !a->z || (a->K > 1 && !a->state) || a->x_stride_b < 0) return KLA_B200_EINVAL;
    if (a->B * a->D > (1ll << 40)) return KLA_B200_EUNSUPPORTED;
    const size_t esz = a->dtype == KLA_B200_F32 ? 4 : 2;
    if (!aligned(a->x, esz) || !aligned(a->z, esz) || (a->state && !aligned(a->state, esz))) return KLA_B200_EALIGN;
    ConvStepParams prm{};
    prm.B = (int)a->B; prm.D = (int)a->D; prm.K = (int)a->K;
    prm.x = a->x; prm.x_sb = a->x_stride_b; prm.w = a->weight; prm.bias = a->bias;
    prm.state = a->state; prm.z = a->z; prm.act = a->activation;
    const unsigned blocks = (unsigned)((a->B * a->D + 127) / 128);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (a->dtype == KLA_B200_F32) kla_conv_step_kernel<float><<<blocks, 128, 0, st>>>(prm);
    else kla_conv_step_kernel<__nv_bfloat16><<<blocks, 128, 0, st>>>(prm);
    g_launches++;
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

int kla_b200_conv_seq(const kla_b200_conv_seq_args *a, void *stream) {
    if (a == nullptr || a->B < 0 || a->L < 0 || a->D < 0) return KLA_B200_EINVAL;
    if (a->K < 1 || a->K > KLA_B200_MAX_CONV_TAPS) return KLA_B200_EUNSUPPORTED;
    if (a->dtype != KLA_B200_F32 && a->dtype != KLA_B200_BF16) return KLA_B200_EUNSUPPORTED;
    if (a->activation < KLA_B200_ACT_SILU || a->activation > KLA_B200_ACT_NONE) return KLA_B200_EINVAL;
    if (a->B > 65535 || a->L > (1 << 30) || a->D > (1 << 30)) return KLA_B200_EUNSUPPORTED;
    if (a->B == 0 || a->D == 0 || a->L == 0) return KLA_B200_OK;
    if (!a->weight || (a->K > 1 && (!a->state || !a->state_out || a->state == a->state_out))) return KLA_B200_EINVAL;
    const size_t esz = a->dtype == KLA_B200_F32 ? 4 : 2;
    int rc;
    if ((rc = check_t3(a->x, esz, true))) return rc;
    if ((rc = check_t3(a->z, esz, true))) return rc;
    if ((a->state && !aligned(a->state, esz)) || (a->state_out && !aligned(a->state_out, esz))) return KLA_B200_EALIGN;
    const int64_t chunks = (a->L + kConvChunk - 1) / kConvChunk;
    if (chunks > 65535) return KLA_B200_EUNSUPPORTED;
    ConvSeqParams prm{};
    prm.B = (int)a->B; prm.L = (int)a->L; prm.D = (int)a->D; prm.K = (int)a->K;
    prm.x = t3(a->x); prm.z = t3(a->z); prm.w = a->weight; prm.bias = a->bias; prm.state = a->state;
    prm.state_out = a->state_out; prm.act = a->activation;
    // two channels per thread when every row starts on a 2-element boundary
    const bool pair = a->D % 2 == 0 && pair_ok(a->x, esz) && pair_ok(a->z, esz);
    const int64_t lanes = pair ? a->D / 2 : a->D;
    dim3 grid((unsigned)((lanes + 127) / 128), (unsigned)chunks, (unsigned)a->B);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define KLA_CONV_LAUNCH(KERNEL, T)                                                    \
    do {                                                                              \
        if (a->K == 4 && a->activation == KLA_B200_ACT_SILU) {                        \
            if (pair) KERNEL<T, 2, 4, true><<<grid, 128, 0, st>>>(prm);               \
            else KERNEL<T, 1, 4, true><<<grid, 128, 0, st>>>(prm);                    \
        } else if (a->K <= 4) {                                                       \
            if (pair) KERNEL<T, 2, 4, false><<<grid, 128, 0, st>>>(prm);              \
            else KERNEL<T, 1, 4, false><<<grid, 128, 0, st>>>(prm);                   \
        } else {                                                                      \
            if (pair) KERNEL<T, 2, kConvMaxTaps, false><<<grid, 128, 0, st>>>(prm);   \
            else KERNEL<T, 1, kConvMaxTaps, false><<<grid, 128, 0, st>>>(prm);        \
        }                                                                             \
    } while (0)
    if (a->dtype == KLA_B200_F32) KLA_CONV_LAUNCH(kla_conv_seq_kernel, float);
    else KLA_CONV_LAUNCH(kla_conv_seq_kernel, __nv_bfloat16);
#undef KLA_CONV_LAUNCH
    g_launches++;
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

int kla_b200_conv_seq_bwd(const kla_b200_conv_seq_bwd_args *a, void *stream) {
    if (a == nullptr || a->B < 0 || a->L < 0 || a->D < 0) return KLA_B200_EINVAL;
    if (a->K < 1 || a->K > KLA_B200_MAX_CONV_TAPS) return KLA_B200_EUNSUPPORTED;
    if (a->dtype != KLA_B200_F32 && a->dtype != KLA_B200_BF16) return KLA_B200_EUNSUPPORTED;
    if (a->activation < KLA_B200_ACT_SILU || a->activation > KLA_B200_ACT_NONE) return KLA_B200_EINVAL;
    if (a->B > 65535 || a->L > (1 << 30) || a->D > (1 << 30)) return KLA_B200_EUNSUPPORTED;
    if (a->B == 0 || a->D == 0 || a->L == 0) return KLA_B200_OK;
    if (!a->weight || !a->dweight) return KLA_B200_EINVAL;
    const size_t esz = a->dtype == KLA_B200_F32 ? 4 : 2;
    int rc;
    if ((rc = check_t3(a->x, esz, true)) || (rc = check_t3(a->dz, esz, true)) || (rc = check_t3(a->dx, esz, true))) return rc;
    if (a->state && !aligned(a->state, esz)) return KLA_B200_EALIGN;
    const int64_t chunks = (a->L + kConvBwdChunk - 1) / kConvBwdChunk;
    if (chunks > 65535) return KLA_B200_EUNSUPPORTED;
    ConvSeqBwdParams prm{};
    prm.B = (int)a->B; prm.L = (int)a->L; prm.D = (int)a->D; prm.K = (int)a->K;
    prm.x = t3(a->x); prm.dz = t3(a->dz); prm.dx = t3(a->dx); prm.w = a->weight; prm.bias = a->bias;
    prm.state = a->state; prm.dw = a->dweight; prm.dbias = a->dbias; prm.act = a->activation;
    // One channel per thread: with two, the backward's register windows cost in occupancy what the wider accesses give
    // back (B=16 L=2048 D=1536 bfloat16 152 against 156 us for the layer's default, 215 against 350 us for other taps).
    dim3 grid((unsigned)((a->D + 127) / 128), (unsigned)chunks, (unsigned)a->B);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define KLA_CONV_BWD_LAUNCH(T)                                                                  \
    do {                                                                                        \
        if (a->K == 4 && a->activation == KLA_B200_ACT_SILU)                                    \
            kla_conv_seq_bwd_kernel<T, 1, 4, true><<<grid, 128, 0, st>>>(prm);                 \
        else if (a->K <= 4) kla_conv_seq_bwd_kernel<T, 1, 4, false><<<grid, 128, 0, st>>>(prm); \
        else kla_conv_seq_bwd_kernel<T, 1, kConvMaxTaps, false><<<grid, 128, 0, st>>>(prm);     \
    } while (0)
    if (a->dtype == KLA_B200_F32) KLA_CONV_BWD_LAUNCH(float);
    else KLA_CONV_BWD_LAUNCH(__nv_bfloat16);
#undef KLA_CONV_BWD_LAUNCH
    g_launches++;
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

int kla_b200_add_norm(int64_t rows, int64_t D, int32_t dtype, int32_t weight_dtype, const void *x, const void *delta, const void *weight,
                      float eps, void *sum, void *out, void *stream) {
    if (rows < 0 || D < 0) return KLA_B200_EINVAL;
    if (D % 8 || D > (1 << 30) || rows > 0x7fffffffll || !known_type(dtype) || !known_type(weight_dtype)) return KLA_B200_EUNSUPPORTED;
    if (rows == 0 || D == 0) return KLA_B200_OK;
    if (!x || !weight || !out || (delta && !sum)) return KLA_B200_EINVAL;
    for (const void *p : {x, delta, weight, static_cast<const void *>(sum), static_cast<const void *>(out)})
        if (p && !aligned(p, 16)) return KLA_B200_EALIGN;
    const AddNormParams prm{(int)rows, (int)D, x, delta, weight, sum, out, eps};
    const unsigned grid = (unsigned)((rows + 3) / 4);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool b = dtype == KLA_B200_BF16, wb = weight_dtype == KLA_B200_BF16;
    if (b && wb) kla_add_norm_kernel<__nv_bfloat16, __nv_bfloat16><<<grid, 128, 0, st>>>(prm);
    else if (b) kla_add_norm_kernel<__nv_bfloat16, float><<<grid, 128, 0, st>>>(prm);
    else if (wb) kla_add_norm_kernel<float, __nv_bfloat16><<<grid, 128, 0, st>>>(prm);
    else kla_add_norm_kernel<float, float><<<grid, 128, 0, st>>>(prm);
    g_launches++;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

int kla_b200_swiglu(int64_t rows, int64_t H, int32_t dtype, const void *gate_up, void *out, void *stream) {
    if (rows < 0 || H < 0) return KLA_B200_EINVAL;
    if (H % 8 || H > (1 << 29) || rows > (1ll << 31) || !known_type(dtype)) return KLA_B200_EUNSUPPORTED;
    if (rows == 0 || H == 0) return KLA_B200_OK;
    if (!gate_up || !out) return KLA_B200_EINVAL;
    if (!aligned(gate_up, 16) || !aligned(out, 16)) return KLA_B200_EALIGN;
    const long long blocks = (rows * (H / 8) + 255) / 256;
    if (blocks > 0x7fffffffll) return KLA_B200_EUNSUPPORTED;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == KLA_B200_BF16)
        kla_swiglu_kernel<<<(unsigned)blocks, 256, 0, st>>>(static_cast<const __nv_bfloat16 *>(gate_up), static_cast<__nv_bfloat16 *>(out), rows, (int)H);
    else
        kla_swiglu_kernel<<<(unsigned)blocks, 256, 0, st>>>(static_cast<const float *>(gate_up), static_cast<float *>(out), rows, (int)H);
    g_launches++;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

int kla_b200_qk_norm(int64_t B, int64_t L, int64_t S, int32_t dtype, kla_b200_tensor3 k, kla_b200_tensor3 q, float clip, void *k_out,
                     void *q_out, void *stream) {
    int rc = check_common(B, L, 1, S, dtype, dtype);
    if (rc) return rc;
    if (B == 0 || L == 0 || S == 0) return KLA_B200_OK;
    const size_t esz = dtype == KLA_B200_F32 ? 4 : 2;
    if (!k_out || !q_out) return KLA_B200_EINVAL;
    if ((rc = check_t3(k, esz, true)) || (rc = check_t3(q, esz, true))) return rc;
    if (!aligned(k_out, esz) || !aligned(q_out, esz)) return KLA_B200_EALIGN;
    const long long blocks = (B * L + 3) / 4;
    if (blocks > 0x7fffffffll) return KLA_B200_EUNSUPPORTED;
    const QkNormParams prm{(int)B, (int)L, (int)S, t3(k), t3(q), k_out, q_out, clip};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (dtype == KLA_B200_BF16) kla_qk_norm_kernel<__nv_bfloat16><<<(unsigned)blocks, 128, 0, st>>>(prm);
    else kla_qk_norm_kernel<float><<<(unsigned)blocks, 128, 0, st>>>(prm);
    g_launches++;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

int kla_b200_argmax(int64_t rows, int64_t n, int32_t dtype, const void *x, int64_t row_stride, int64_t *out, void *stream) {
    if (rows < 0 || n < 1 || row_stride < 0) return KLA_B200_EINVAL;
    if (n > (1 << 30) || rows > 0x7fffffffll || !known_type(dtype)) return KLA_B200_EUNSUPPORTED;
    if (rows == 0) return KLA_B200_OK;
    if (!x || !out) return KLA_B200_EINVAL;
    if (!aligned(x, dtype == KLA_B200_BF16 ? 2 : 4) || !aligned(out, 8)) return KLA_B200_EALIGN;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    long long *o = reinterpret_cast<long long *>(out);
    if (dtype == KLA_B200_BF16) kla_argmax_kernel<<<(unsigned)rows, 1024, 0, st>>>(static_cast<const __nv_bfloat16 *>(x), row_stride, (int)n, o);
    else kla_argmax_kernel<<<(unsigned)rows, 1024, 0, st>>>(static_cast<const float *>(x), row_stride, (int)n, o);
    g_launches++;
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? KLA_B200_OK : cuda_fail(e);
}

int kla_b200_linear(const kla_b200_linear_args *a, void *stream) {
    if (a == nullptr || a->B < 0 || a->N < 0 || a->K < 0) return KLA_B200_EINVAL;
    if (a->B > KLA_B200_LINEAR_MAX_ROWS || a->N > (1 << 30) || a->K > (1 << 20) || a->K % 8 || a->x_stride_b % 8) return KLA_B200_EUNSUPPORTED;
    if (a->B == 0 || a->N == 0) return KLA_B200_OK;
    if (a->K == 0 || !a->x || !a->weight || !a->out || a->x_stride_b < 0 || a->out_stride_b < 0 || a->residual_stride_b < 0) return KLA_B200_EINVAL;
    for (const void *p : {a->x, a->weight, a->norm_weight})
        if (p && !aligned(p, 16)) return KLA_B200_EALIGN;
    for (const void *p : {a->bias, a->residual, static_cast<const void *>(a->out), static_cast<const void *>(a->conv_state)})
        if (p && !aligned(p, 2)) return KLA_B200_EALIGN;
    if (a->swiglu && (a->N % 2 || a->conv_D)) return KLA_B200_EINVAL;
    LinearParams prm{};
    prm.B = (int)a->B; prm.N = (int)a->N; prm.K = (int)a->K;
    prm.x = static_cast<const __nv_bfloat16 *>(a->x); prm.x_sb = a->x_stride_b;
    prm.w = static_cast<const __nv_bfloat16 *>(a->weight); prm.bias = static_cast<const __nv_bfloat16 *>(a->bias);
    prm.out = static_cast<__nv_bfloat16 *>(a->out); prm.out_sb = a->out_stride_b;
    prm.norm_w = static_cast<const __nv_bfloat16 *>(a->norm_weight); prm.norm_eps = a->norm_eps;
    prm.res = static_cast<const __nv_bfloat16 *>(a->residual); prm.res_sb = a->residual_stride_b;
    if (a->conv_D) {
        if (a->conv_D < 0 || a->conv_D > a->N || a->conv_taps < 1 || a->conv_taps > KLA_B200_MAX_CONV_TAPS) return KLA_B200_EUNSUPPORTED;
        if (!a->conv_weight || (a->conv_taps > 1 && !a->conv_state)) return KLA_B200_EINVAL;
        if (a->conv_activation < KLA_B200_ACT_SILU || a->conv_activation > KLA_B200_ACT_NONE) return KLA_B200_EINVAL;
        prm.D = (int)a->conv_D; prm.taps = (int)a->conv_taps; prm.conv_act = a->conv_activation;
        prm.conv_w = a->conv_weight; prm.conv_b = a->conv_bias; prm.conv_state = static_cast<__nv_bfloat16 *>(a->conv_state);
    }
    prm.weights_ready = a->weights_ready;
    const int mode = a->swiglu ? kLinearSwiglu : a->conv_D ? kLinearConv : kLinearPlain;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (a->B <= 8) return dispatch_linear<1>(prm, mode, st);
    if (a->B <= 16) return dispatch_linear<2>(prm, mode, st);
    return dispatch_linear<4>(prm, mode, st);
}

size_t kla_b200_token_work_bytes(const kla_b200_token_args *a) { return check_token(a) == KLA_B200_OK ? token_work(a).total : 0; }

int kla_b200_token(const kla_b200_token_args *a, void *stream) {
    if (int rc = check_token(a)) return rc;
    if (a->B == 0 || a->d == 0 || a->layers == 0) return KLA_B200_OK;
    if (!a->x || !a->out || !a->work || a->x_stride_b < 0 || (a->y_var && a->layers != 1)) return KLA_B200_EINVAL;
    if (a->x_stride_b % 8) return KLA_B200_EUNSUPPORTED;
    if (!aligned(a->x, 16) || !aligned(a->out, 16) || !aligned(a->work, 256) || !aligned(a->y_var, 2)) return KLA_B200_EALIGN;
    for (int64_t i = 0; i < a->layers; ++i) {
        const kla_b200_token_layer &l = a->layer[i];
        if (!l.in_weight || !l.sensor_weight || !l.out_weight || !l.a || !l.p || !l.lam || !l.eta) return KLA_B200_EINVAL;
        if ((a->mlp && (!l.w12 || !l.w3 || !l.mlp_norm_weight)) || (l.conv_weight && l.conv_taps > 1 && !l.conv_state) || (l.lambda_skip_len && !l.lambda_skip))
            return KLA_B200_EINVAL;
        for (const void *p : {l.in_weight, l.sensor_weight, l.out_weight, l.norm_weight, a->mlp ? l.w12 : nullptr, a->mlp ? l.w3 : nullptr, a->mlp ? l.mlp_norm_weight : nullptr})
            if (p && !aligned(p, 16)) return KLA_B200_EALIGN;
        for (const void *p : {l.in_bias, l.sensor_bias, l.out_bias, l.b12, l.b3, static_cast<const void *>(l.conv_state)})
            if (p && !aligned(p, 2)) return KLA_B200_EALIGN;
        for (const float *p : {l.conv_weight, l.conv_bias, l.a, l.p, l.lambda_skip, static_cast<const float *>(l.lam), static_cast<const float *>(l.eta)})
            if (p && !aligned(p, 4)) return KLA_B200_EALIGN;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return a->layers == 1 ? launch_token<1>(a, st) : launch_token<KLA_B200_TOKEN_MAX_LAYERS>(a, st);
}

int kla_b200_step_layer(const kla_b200_step_layer_args *a, void *stream) {
    if (a == nullptr) return KLA_B200_EINVAL;
    int rc = check_common(a->B, 1, a->M, a->S, a->in_dtype, a->out_dtype);
    if (rc) return rc;
    if (a->gate_activation < KLA_B200_ACT_SILU || a->gate_activation > KLA_B200_ACT_NONE) return KLA_B200_EINVAL;
    if (a->lambda_skip_len != 0 && a->lambda_skip_len != 1 && a->lambda_skip_len != a->M) return KLA_B200_EINVAL;
    if (a->B == 0 || a->M == 0) return KLA_B200_OK;
    if (!a->v || !a->log_sigma_v || !a->y || !a->y_var || !a->a || !a->p) return KLA_B200_EINVAL;
    if (a->S > 0 && (!a->k || !a->q || !a->lam || !a->eta || !a->lam_out || !a->eta_out)) return KLA_B200_EINVAL;
    if (a->lambda_skip_len != 0 && (!a->lambda_skip || !a->z)) return KLA_B200_EINVAL;
    const size_t esz = a->in_dtype == KLA_B200_F32 ? 4 : 2, osz = a->out_dtype == KLA_B200_F32 ? 4 : 2;
    const void *ps[] = {a->v, a->log_sigma_v, a->k, a->q, a->z, a->gate};
    for (const void *p : ps)
        if (p && !aligned(p, esz)) return KLA_B200_EALIGN;
    if (!aligned(a->y, osz) || !aligned(a->y_var, osz)) return KLA_B200_EALIGN;
    StepLayerParams prm{};
    prm.B = (int)a->B; prm.M = (int)a->M; prm.S = (int)a->S;
    prm.v = a->v; prm.ls = a->log_sigma_v; prm.k = a->k; prm.q = a->q;
    prm.z = a->lambda_skip_len != 0 ? a->z : nullptr; prm.gate = a->gate;
    prm.v_sb = a->v_stride_b; prm.ls_sb = a->log_sigma_v_stride_b; prm.k_sb = a->k_stride_b; prm.q_sb = a->q_stride_b;
    prm.z_sb = a->z_stride_b; prm.gate_sb = a->gate_stride_b;
    prm.a = a->a; prm.p = a->p; prm.lam = a->lam; prm.eta = a->eta;
    prm.lam_out = a->lam_out; prm.eta_out = a->eta_out; prm.y = a->y; prm.yv = a->y_var;
    prm.skip = a->lambda_skip_len != 0 ? a->lambda_skip : nullptr; prm.skip_len = a->lambda_skip_len;
    prm.obs_var_min = a->obs_var_min; prm.obs_var_max = a->obs_var_max; prm.clip = a->clip_value;
    prm.weights_ready = a->weights_ready;
    prm.qk_norm = a->qk_norm; prm.gate_act = a->gate_activation;
    prm.vec = a->S % 4 == 0 && aligned(a->lam, 16) && aligned(a->eta, 16) && aligned(a->a, 16) && aligned(a->p, 16) &&
              aligned(a->lam_out, 16) && aligned(a->eta_out, 16);
    int lpc = 1;
    while (lpc * 4 < a->S) lpc *= 2;
    return dispatch_step_layer(a->in_dtype, a->out_dtype, a->decode_from_prior != 0, lpc, prm, static_cast<cudaStream_t>(stream));
}

const char *kla_b200_strerror(int code) {
    switch (code) {
        case KLA_B200_OK: return "ok";
        case KLA_B200_EINVAL: return "invalid argument (NULL pointer, negative size or stride, or half of a pointer pair missing)";
        case KLA_B200_EUNSUPPORTED: return "unsupported configuration (d_state above 128, unsupported dtype pair, or a dimension too large)";
        case KLA_B200_EALIGN: return "pointer not aligned to its element size";
        case KLA_B200_ETOOBIG: return "problem too large for the library's built-in checkpoint scratch (KLA_B200_STATIC_CKPT_BYTES); use kla_b200_scan_fwd with caller-provided scratch";
        case KLA_B200_ECUDA:
            snprintf(g_errbuf, sizeof(g_errbuf), "CUDA error: %s", cudaGetErrorString(g_last_cuda));
            return g_errbuf;
        default: return "unknown error code";
    }
}

int kla_b200_version(void) { return 100; }

int64_t kla_b200_launch_count(void) { return g_launches.load(); }

// ---------------------------------------------------------------------------
// Forward scan with its checkpoint scratch inside the library.
//
// The scratch is a fixed array in device memory that every GPU loading this
// library carries until the process exits. In host code the name of a
// __device__ array is only a handle, not an address a kernel can use, so the
// device address is looked up once per device with cudaGetSymbolAddress and
// cached here.
static __device__ __align__(256) unsigned char g_static_ckpt[KLA_B200_STATIC_CKPT_BYTES];

namespace {
std::mutex g_static_mu;
void *g_static_ckpt_ptr[kMaxDevices] = {};

// Device address of g_static_ckpt on the current device (set up on first use).
int static_ckpt_address(void **out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e);
    if (dev < 0 || dev >= kMaxDevices) return KLA_B200_EUNSUPPORTED;
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (g_static_ckpt_ptr[dev] == nullptr) {
        void *ptr = nullptr;
        e = cudaGetSymbolAddress(&ptr, g_static_ckpt);
        if (e != cudaSuccess) return cuda_fail(e);
        g_static_ckpt_ptr[dev] = ptr;
    }
    *out = g_static_ckpt_ptr[dev];
    return KLA_B200_OK;
}
}  // namespace

int kla_b200_scan_fwd_static(const kla_b200_fwd_args *args, void *stream, const void **ckpt) {
    if (args == nullptr || ckpt == nullptr) return KLA_B200_EINVAL;
    *ckpt = nullptr;
    int rc = check_common(args->B, args->L, args->M, args->S, args->in_dtype, args->out_dtype);
    if (rc) return rc;
    ChunkCtl chunk;  // a cut sequence keeps checkpoints per chunk, more of them than the uncut one
    if ((rc = check_chunks(args->B, args->L, args->chunks, args->chunk_len, &chunk))) return rc;
    if (kla_b200_ckpt_bytes(args->B * chunk.n, chunk.len, args->M, args->S) > (size_t)KLA_B200_STATIC_CKPT_BYTES) return KLA_B200_ETOOBIG;
    void *scratch = nullptr;
    if ((rc = static_ckpt_address(&scratch))) return rc;
    kla_b200_fwd_args a = *args;
    a.ckpt = scratch;  // whatever the caller put there is ignored
    rc = kla_b200_scan_fwd(&a, stream);
    if (rc == KLA_B200_OK) *ckpt = scratch;
    return rc;
}

int kla_b200_mobius_scan_fwd(const kla_b200_rawscan_args *a, void *stream) {
    return launch_rawscan<MobiusFwd>(a, stream, true, false);
}
int kla_b200_mobius_scan_bwd(const kla_b200_rawscan_args *a, void *stream) {
    return launch_rawscan<MobiusBwd>(a, stream, true, true);
}
int kla_b200_affine_scan_fwd(const kla_b200_rawscan_args *a, void *stream) {
    return launch_rawscan<AffineFwd>(a, stream, false, false);
}
int kla_b200_affine_scan_bwd(const kla_b200_rawscan_args *a, void *stream) {
    return launch_rawscan<AffineBwd>(a, stream, false, false);
}

int kla_b200_device_status(int *status) {
    if (status == nullptr) return KLA_B200_EINVAL;
    int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(status, g_kla_status, sizeof(int));
    if (e != cudaSuccess) return cuda_fail(e);
    if (*status != 0) {
        e = cudaMemcpyToSymbol(g_kla_status, &zero, sizeof(int));
        if (e != cudaSuccess) return cuda_fail(e);
    }
    return KLA_B200_OK;
}

int kla_b200_test_hooks(int64_t wait_limit_ns, int32_t skip_tile) {
    if (wait_limit_ns < 0 || wait_limit_ns > 4000000000ll) return KLA_B200_EINVAL;
    g_wait_limit_ns.store(wait_limit_ns == 0 ? 1000000000u : (unsigned)wait_limit_ns);
    g_skip_tile.store(skip_tile < 0 ? -1 : skip_tile);
    return KLA_B200_OK;
}

}  // extern "C"
