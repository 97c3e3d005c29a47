// Native half of the Python wrappers: argument structures, output allocations and launches of the C-ABI library
// (include/kla_b200.h) on torch tensors, one Python call per operation. Filling the structures through ctypes and
// allocating from Python cost 25-40 us per launch, more than most of these kernels run: a decode step of 2.5 us of GPU
// time took 30 us, a small training step of 220 us took 500 us.
//
// The module holds no state but the library's entry points, which bind() receives as addresses, so that it uses the very
// library the Python side loaded. Every function here takes tensors the wrappers have found canonical (same device, dtypes
// and unit last strides checked); canonical() and step() do that check themselves and answer "not this route" otherwise,
// which sends the wrapper to its general path with its error messages.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/kla_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

struct Entry {
    int (*scan_fwd)(const kla_b200_fwd_args *, void *) = nullptr;
    int (*scan_bwd)(const kla_b200_bwd_args *, void *) = nullptr;
    int (*slab_aggregate)(const kla_b200_slab_args *, void *) = nullptr;
    int (*chunk_fold)(const kla_b200_chunk_fold_args *, void *) = nullptr;
    int (*epilogue_bwd)(const kla_b200_epilogue_bwd_args *, void *) = nullptr;
    int (*step)(const kla_b200_step_args *, void *) = nullptr;
    int (*conv_step)(const kla_b200_conv_step_args *, void *) = nullptr;
    int (*step_layer)(const kla_b200_step_layer_args *, void *) = nullptr;
    int (*linear)(const kla_b200_linear_args *, void *) = nullptr;
    size_t (*token_work_bytes)(const kla_b200_token_args *) = nullptr;
    int (*token)(const kla_b200_token_args *, void *) = nullptr;
    int (*add_norm)(int64_t, int64_t, int32_t, int32_t, const void *, const void *, const void *, float, void *, void *, void *) = nullptr;
    int (*swiglu)(int64_t, int64_t, int32_t, const void *, void *, void *) = nullptr;
    int (*qk_norm)(int64_t, int64_t, int64_t, int32_t, kla_b200_tensor3, kla_b200_tensor3, float, void *, void *, void *) = nullptr;
    int (*argmax)(int64_t, int64_t, int32_t, const void *, int64_t, int64_t *, void *) = nullptr;
    int (*conv_seq)(const kla_b200_conv_seq_args *, void *) = nullptr;
    int (*conv_seq_bwd)(const kla_b200_conv_seq_bwd_args *, void *) = nullptr;
    int (*rawscan[4])(const kla_b200_rawscan_args *, void *) = {};  // Moebius forward, backward, affine forward, backward
    size_t (*ckpt_bytes)(int64_t, int64_t, int64_t, int64_t) = nullptr;
    size_t (*segment_scratch_bytes)(int64_t, int64_t, int64_t) = nullptr;
    const char *(*strerror)(int) = nullptr;
} lib;

template <typename F>
void take(F &f, const py::dict &d, const char *name) {
    f = reinterpret_cast<F>(d[name].cast<uintptr_t>());
}

void bind(const py::dict &d) {
    take(lib.scan_fwd, d, "kla_b200_scan_fwd");
    take(lib.scan_bwd, d, "kla_b200_scan_bwd");
    take(lib.slab_aggregate, d, "kla_b200_slab_aggregate");
    take(lib.chunk_fold, d, "kla_b200_chunk_fold");
    take(lib.epilogue_bwd, d, "kla_b200_epilogue_bwd");
    take(lib.step, d, "kla_b200_step");
    take(lib.conv_step, d, "kla_b200_conv_step");
    take(lib.step_layer, d, "kla_b200_step_layer");
    take(lib.linear, d, "kla_b200_linear");
    take(lib.token_work_bytes, d, "kla_b200_token_work_bytes");
    take(lib.token, d, "kla_b200_token");
    take(lib.add_norm, d, "kla_b200_add_norm");
    take(lib.swiglu, d, "kla_b200_swiglu");
    take(lib.qk_norm, d, "kla_b200_qk_norm");
    take(lib.argmax, d, "kla_b200_argmax");
    take(lib.conv_seq, d, "kla_b200_conv_seq");
    take(lib.conv_seq_bwd, d, "kla_b200_conv_seq_bwd");
    take(lib.rawscan[0], d, "kla_b200_mobius_scan_fwd");
    take(lib.rawscan[1], d, "kla_b200_mobius_scan_bwd");
    take(lib.rawscan[2], d, "kla_b200_affine_scan_fwd");
    take(lib.rawscan[3], d, "kla_b200_affine_scan_bwd");
    take(lib.ckpt_bytes, d, "kla_b200_ckpt_bytes");
    take(lib.segment_scratch_bytes, d, "kla_b200_segment_scratch_bytes");
    take(lib.strerror, d, "kla_b200_strerror");
}

// The C-ABI status as the exception the Python side's _lib.check raises for it.
void check(int rc) {
    if (rc == KLA_B200_OK) return;
    const std::string msg = lib.strerror(rc);
    if (rc == KLA_B200_EUNSUPPORTED) {
        PyErr_SetString(PyExc_NotImplementedError, ("The b200 KLA backend: " + msg + ". Use backend='torch' for this case.").c_str());
        throw py::error_already_set();
    }
    if (rc == KLA_B200_EINVAL || rc == KLA_B200_EALIGN || rc == KLA_B200_ETOOBIG) throw py::value_error("kla_b200: " + msg);
    throw std::runtime_error("kla_b200: " + msg);
}

// Tensors the kernels would read or write past their end, or as another type.
void require(bool ok, const char *what) {
    if (!ok) throw py::value_error(std::string("kla_b200: ") + what);
}
void require_type(const Tensor &t) {
    const auto T = t.scalar_type();
    if (T == at::kFloat || T == at::kBFloat16) return;
    PyErr_SetString(PyExc_NotImplementedError, (std::string("The b200 kernels take float32 or bfloat16 activations, not ") + c10::toString(T) + ".").c_str());
    throw py::error_already_set();
}
bool is(const Tensor &t, const at::Device &dev, at::ScalarType type, at::IntArrayRef sizes) {
    return t.device() == dev && t.scalar_type() == type && t.sizes() == sizes && t.is_contiguous();
}

kla_b200_tensor3 t3(const Tensor &t) { return kla_b200_tensor3{t.data_ptr(), t.stride(0), t.stride(1)}; }
kla_b200_tensor3 t3(const OptTensor &t) { return t ? t3(*t) : kla_b200_tensor3{nullptr, 0, 0}; }
float *fp(const Tensor &t) { return static_cast<float *>(t.data_ptr()); }
float *fp(const OptTensor &t) { return t ? fp(*t) : nullptr; }
int32_t dt(at::ScalarType t) { return t == at::kBFloat16 ? KLA_B200_BF16 : KLA_B200_F32; }
at::ScalarType out_type(bool bf16) { return bf16 ? at::kBFloat16 : at::kFloat; }
void *stream_of(const Tensor &t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
// An uninitialised contiguous tensor on like's device, straight from the CUDA allocator (no dispatch).
Tensor fresh(const Tensor &like, at::IntArrayRef sizes, at::ScalarType type) {
    return Tensor(at::detail::empty_cuda(sizes, type, like.device(), std::nullopt));
}
Tensor fresh(const Tensor &like, at::IntArrayRef sizes) { return fresh(like, sizes, like.scalar_type()); }
Tensor f32(const Tensor &like, at::IntArrayRef sizes) { return fresh(like, sizes, at::kFloat); }

struct Sensors {
    bool on = false;
    float vmin = 0.0f, vmax = 0.0f;
    explicit Sensors(const std::optional<std::tuple<double, std::optional<double>>> &s) {
        if (!s) return;
        on = true;
        vmin = (float)std::get<0>(*s);
        vmax = (float)std::get<1>(*s).value_or(0.0);
    }
};
using SensorArg = std::optional<std::tuple<double, std::optional<double>>>;

bool rows_ok(const Tensor &t) { return t.size(-1) <= 1 || t.stride(-1) == 1; }
bool sm100(const at::Device &d) { return at::cuda::getDeviceProperties(d.index())->major == 10; }

// Whether the scan's arguments need no conversion, copy or error message.
bool canonical(const Tensor &v, const Tensor &lv, const Tensor &k, const Tensor &q, const Tensor &a, const Tensor &p,
               const OptTensor &lam0, const OptTensor &eta0) {
    if (!v.is_cuda() || v.dim() != 3 || k.dim() != 3 || a.dim() != 2) return false;
    const auto T = v.scalar_type();
    if (T != at::kFloat && T != at::kBFloat16) return false;
    if (lv.scalar_type() != T || k.scalar_type() != T || q.scalar_type() != T) return false;
    if (a.scalar_type() != at::kFloat || p.scalar_type() != at::kFloat || !a.is_contiguous() || !p.is_contiguous()) return false;
    const int64_t B = v.size(0), L = v.size(1), M = v.size(2), S = k.size(2);
    if (S > KLA_B200_MAX_DSTATE || lv.sizes() != v.sizes() || q.sizes() != k.sizes() || k.size(0) != B || k.size(1) != L) return false;
    if (a.size(0) != M || a.size(1) != S || p.sizes() != a.sizes()) return false;
    const auto dev = v.device();
    if (lv.device() != dev || k.device() != dev || q.device() != dev || a.device() != dev || p.device() != dev) return false;
    if (!rows_ok(v) || !rows_ok(lv) || !rows_ok(k) || !rows_ok(q)) return false;
    if (lam0.has_value() != eta0.has_value()) return false;
    if (lam0) {
        for (const Tensor *t : {&*lam0, &*eta0})
            if (t->scalar_type() != at::kFloat || !t->is_contiguous() || t->device() != dev || t->dim() != 3 || t->size(0) != B ||
                t->size(1) != M || t->size(2) != S)
                return false;
    }
    return sm100(dev);
}

// ------------------------------------------------------------------------------------------------------ the scan

// kla_b200_scan_fwd. segments: give the kernel working memory so that a forward without checkpoints can hand sequences
// from CTA to CTA. chunks > 1: lam0 and eta0 are per chunk.
std::tuple<Tensor, Tensor, Tensor, Tensor, OptTensor> scan_fwd(
    const Tensor &v, const Tensor &lv, const Tensor &k, const Tensor &q, const Tensor &a, const Tensor &p, const OptTensor &lam0,
    const OptTensor &eta0, bool prior, bool out_bf16, bool need_ckpt, bool segments, const SensorArg &sensors, const OptTensor &z,
    const OptTensor &skip, const OptTensor &gate, int gate_act, const OptTensor &y_raw, const OptTensor &yv_raw, int64_t chunks,
    int64_t chunk_len) {
    const c10::cuda::CUDAGuard guard(v.device());
    const int64_t B = v.size(0), L = v.size(1), M = v.size(2), S = k.size(2), E = B * chunks;
    const auto TO = out_type(out_bf16);
    Tensor y = fresh(v, {B, L, M}, TO), yv = fresh(v, {B, L, M}, TO);
    Tensor lam = f32(v, {B, M, S}), eta = f32(v, {B, M, S});
    OptTensor ckpt, work;
    if (need_ckpt && L > 0) ckpt = fresh(v, {(int64_t)lib.ckpt_bytes(E, chunks > 1 ? chunk_len : L, M, S)}, at::kByte);
    else if (segments) work = fresh(v, {(int64_t)lib.segment_scratch_bytes(B, M, S)}, at::kByte);
    const Sensors sen(sensors);
    kla_b200_fwd_args f{};
    f.B = B; f.L = L; f.M = M; f.S = S;
    f.in_dtype = dt(v.scalar_type()); f.out_dtype = dt(TO); f.decode_from_prior = prior;
    f.v = t3(v); f.lambda_v = t3(lv); f.k = t3(k); f.q = t3(q);
    f.a = fp(a); f.p = fp(p); f.lam0 = fp(lam0); f.eta0 = fp(eta0);
    f.y = t3(y); f.y_var = t3(yv); f.lam_fin = fp(lam); f.eta_fin = fp(eta);
    f.ckpt = ckpt ? ckpt->data_ptr() : nullptr;
    f.work = work ? work->data_ptr() : nullptr;
    f.lambda_v_is_log_variance = sen.on; f.obs_var_min = sen.vmin; f.obs_var_max = sen.vmax;
    if (skip) { f.z = t3(z); f.lambda_skip = fp(*skip); f.lambda_skip_len = (int32_t)skip->numel(); }
    if (gate) { f.gate = t3(*gate); f.gate_activation = gate_act; }
    f.y_raw = t3(y_raw); f.y_var_raw = t3(yv_raw);
    if (chunks > 1) { f.chunks = chunks; f.chunk_len = chunk_len; f.sequence_state = 1; }
    check(lib.scan_fwd(&f, stream_of(v)));
    return {y, yv, lam, eta, ckpt};
}

// kla_b200_scan_bwd -> dv, dlambda_v, dk, dq, da, dp, dlam0, deta0
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> scan_bwd(
    const Tensor &v, const Tensor &lv, const Tensor &k, const Tensor &q, const Tensor &a, const Tensor &p, const OptTensor &lam0,
    const OptTensor &eta0, const OptTensor &ckpt, const Tensor &dy, const OptTensor &dyv, const OptTensor &dlam_fin,
    const OptTensor &deta_fin, bool prior, bool out_bf16, const SensorArg &sensors, int64_t chunks, int64_t chunk_len) {
    const c10::cuda::CUDAGuard guard(v.device());
    const int64_t B = v.size(0), L = v.size(1), M = v.size(2), S = k.size(2), E = B * chunks;
    Tensor dv = fresh(v, {B, L, M}), dlv = fresh(v, {B, L, M});
    Tensor dk = f32(v, {B, L, S}), dq = f32(v, {B, L, S}), da = f32(v, {M, S}), dp = f32(v, {M, S});
    Tensor dlam0 = f32(v, {E, M, S}), deta0 = f32(v, {E, M, S});
    const Sensors sen(sensors);
    kla_b200_bwd_args b{};
    b.B = B; b.L = L; b.M = M; b.S = S;
    b.in_dtype = dt(v.scalar_type()); b.out_dtype = out_bf16 ? KLA_B200_BF16 : KLA_B200_F32; b.decode_from_prior = prior;
    b.v = t3(v); b.lambda_v = t3(lv); b.k = t3(k); b.q = t3(q);
    b.a = fp(a); b.p = fp(p); b.lam0 = fp(lam0); b.eta0 = fp(eta0);
    b.ckpt = ckpt ? ckpt->data_ptr() : nullptr;
    b.dy = t3(dy); b.dy_var = t3(dyv); b.dlam_fin = fp(dlam_fin); b.deta_fin = fp(deta_fin);
    b.dv = t3(dv); b.dlambda_v = t3(dlv); b.dk = fp(dk); b.dq = fp(dq); b.da = fp(da); b.dp = fp(dp);
    b.dlam0 = fp(dlam0); b.deta0 = fp(deta0);
    b.lambda_v_is_log_variance = sen.on; b.obs_var_min = sen.vmin; b.obs_var_max = sen.vmax;
    if (chunks > 1) { b.chunks = chunks; b.chunk_len = chunk_len; }
    check(lib.scan_bwd(&b, stream_of(v)));
    return {dv, dlv, dk, dq, da, dp, dlam0, deta0};
}

// kla_b200_slab_aggregate -> [B*chunks, M, S, 8]; the adjoint aggregate when dy is given
Tensor slab_aggregate(const Tensor &v, const Tensor &lv, const Tensor &k, const Tensor &a, const Tensor &p, const OptTensor &q,
                      const OptTensor &dy, const OptTensor &dyv, const OptTensor &lam0, const OptTensor &eta0, bool prior,
                      const SensorArg &sensors, int64_t chunks, int64_t chunk_len) {
    const c10::cuda::CUDAGuard guard(v.device());
    const int64_t B = v.size(0), L = v.size(1), M = v.size(2), S = k.size(2);
    Tensor out = f32(v, {B * chunks, M, S, 8});
    kla_b200_slab_args s{};
    s.B = B; s.L = L; s.M = M; s.S = S;
    s.in_dtype = dt(v.scalar_type()); s.out_dtype = dy ? dt(dy->scalar_type()) : KLA_B200_F32;
    s.decode_from_prior = prior; s.adjoint = dy.has_value();
    s.v = t3(v); s.lambda_v = t3(lv); s.k = t3(k); s.q = t3(q);
    s.a = fp(a); s.p = fp(p); s.lam0 = fp(lam0); s.eta0 = fp(eta0);
    s.dy = t3(dy); s.dy_var = t3(dyv); s.out = fp(out);
    const Sensors sen(sensors);
    s.lambda_v_is_log_variance = sen.on; s.obs_var_min = sen.vmin; s.obs_var_max = sen.vmax;
    if (chunks > 1) { s.chunks = chunks; s.chunk_len = chunk_len; }
    check(lib.slab_aggregate(&s, stream_of(v)));
    return out;
}

// kla_b200_chunk_fold over aggregates [B*C, M, S, 8] -> two [B*C, M, S]
std::tuple<Tensor, Tensor> chunk_fold(const Tensor &agg, int64_t C, const OptTensor &in_a, const OptTensor &in_b, const OptTensor &lam_in,
                                      const OptTensor &eta_in, bool adjoint) {
    const c10::cuda::CUDAGuard guard(agg.device());
    const int64_t E = agg.size(0), M = agg.size(1), S = agg.size(2);
    Tensor out_a = f32(agg, {E, M, S}), out_b = f32(agg, {E, M, S});
    kla_b200_chunk_fold_args c{};
    c.B = E / C; c.C = C; c.M = M; c.S = S; c.adjoint = adjoint;
    c.agg = fp(agg); c.in_a = fp(in_a); c.in_b = fp(in_b); c.lam_in = fp(lam_in); c.eta_in = fp(eta_in); c.out_a = fp(out_a); c.out_b = fp(out_b);
    check(lib.chunk_fold(&c, stream_of(agg)));
    return {out_a, out_b};
}

// The time-parallel forward: aggregates, fold, scan over the chunks. -> y, y_var, the sequences' final state, the
// checkpoints and every chunk's start state (both for the backward).
std::tuple<Tensor, Tensor, Tensor, Tensor, OptTensor, Tensor, Tensor> scan_fwd_chunked(
    const Tensor &v, const Tensor &lv, const Tensor &k, const Tensor &q, const Tensor &a, const Tensor &p, const OptTensor &lam0,
    const OptTensor &eta0, bool prior, bool out_bf16, bool need_ckpt, const SensorArg &sensors, const OptTensor &z,
    const OptTensor &skip, const OptTensor &gate, int gate_act, const OptTensor &y_raw, const OptTensor &yv_raw, int64_t chunks,
    int64_t chunk_len) {
    const Tensor agg = slab_aggregate(v, lv, k, a, p, {}, {}, {}, {}, {}, false, sensors, chunks, chunk_len);
    auto [lam_in, eta_in] = chunk_fold(agg, chunks, lam0, eta0, {}, {}, false);
    auto [y, yv, lam, eta, ckpt] = scan_fwd(v, lv, k, q, a, p, lam_in, eta_in, prior, out_bf16, need_ckpt, false, sensors, z, skip,
                                            gate, gate_act, y_raw, yv_raw, chunks, chunk_len);
    return {y, yv, lam, eta, ckpt, lam_in, eta_in};
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> scan_bwd_chunked(
    const Tensor &v, const Tensor &lv, const Tensor &k, const Tensor &q, const Tensor &a, const Tensor &p, const Tensor &lam_in,
    const Tensor &eta_in, const OptTensor &ckpt, const Tensor &dy, const OptTensor &dyv, const OptTensor &dlam_fin,
    const OptTensor &deta_fin, bool prior, bool out_bf16, const SensorArg &sensors, int64_t chunks, int64_t chunk_len) {
    const Tensor agg = slab_aggregate(v, lv, k, a, p, q, dy, dyv, lam_in, eta_in, prior, sensors, chunks, chunk_len);
    auto [dlam_seed, deta_seed] = chunk_fold(agg, chunks, dlam_fin, deta_fin, lam_in, eta_in, true);
    auto r = scan_bwd(v, lv, k, q, a, p, lam_in, eta_in, ckpt, dy, dyv, dlam_seed, deta_seed, prior, out_bf16, sensors, chunks, chunk_len);
    const int64_t B = v.size(0), M = v.size(2), S = k.size(2);
    auto first = [&](const Tensor &t) { return t.view({B, chunks, M, S}).select(1, 0); };
    std::get<6>(r) = first(std::get<6>(r));
    std::get<7>(r) = first(std::get<7>(r));
    return r;
}

// kla_b200_epilogue_bwd -> dy, dy_var for the scan's backward, and dz, dgate, dskip of the halves that are there
std::tuple<Tensor, Tensor, OptTensor, OptTensor, OptTensor> epilogue_bwd(const Tensor &v, bool out_bf16, const Tensor &dout,
                                                                        const OptTensor &dout_var, const OptTensor &y_raw,
                                                                        const OptTensor &yv_raw, const OptTensor &z,
                                                                        const OptTensor &gate, const OptTensor &skip, int gate_act) {
    const c10::cuda::CUDAGuard guard(v.device());
    const int64_t B = v.size(0), L = v.size(1), M = v.size(2);
    const auto TO = out_type(out_bf16);
    Tensor dy = fresh(v, {B, L, M}, TO), dyv = fresh(v, {B, L, M}, TO);
    OptTensor dz, dgate, dskip, work;
    if (z) dz = fresh(v, {B, L, M});
    if (gate) dgate = fresh(v, {B, L, M});
    if (skip) dskip = at::empty_like(*skip);
    if (skip && skip->numel() == 1) work = fresh(v, {KLA_B200_SKIP_SUM_BYTES}, at::kByte);
    kla_b200_epilogue_bwd_args e{};
    e.B = B; e.L = L; e.M = M;
    e.in_dtype = dt(v.scalar_type()); e.out_dtype = dt(TO);
    e.gate_activation = gate ? gate_act : KLA_B200_ACT_NONE;
    e.lambda_skip_len = skip ? (int32_t)skip->numel() : 0;
    e.dout = t3(dout); e.dout_var = t3(dout_var); e.y_raw = t3(y_raw); e.y_var_raw = t3(yv_raw);
    e.z = t3(z); e.gate = t3(gate); e.lambda_skip = fp(skip);
    e.dy = t3(dy); e.dy_var = t3(dyv); e.dz = t3(dz); e.dgate = t3(dgate); e.dlambda_skip = fp(dskip);
    e.work = work ? work->data_ptr() : nullptr;
    check(lib.epilogue_bwd(&e, stream_of(v)));
    return {dy, dyv, dz, dgate, dskip};
}

// kla_b200_conv_seq -> z, the window after the sequence
std::tuple<Tensor, Tensor> conv_seq(const Tensor &x, const Tensor &w, const OptTensor &bias, const Tensor &state, int act) {
    const c10::cuda::CUDAGuard guard(x.device());
    require_type(x);
    require(x.dim() == 3 && w.dim() == 2 && w.size(0) == x.size(2) && w.size(1) >= 1, "the convolution takes x [B, L, D] and weights [D, K]");
    const int64_t B = x.size(0), L = x.size(1), D = x.size(2);
    require(rows_ok(x) && is(w, x.device(), at::kFloat, w.sizes()) && (!bias || is(*bias, x.device(), at::kFloat, {D})) &&
                is(state, x.device(), x.scalar_type(), {B, D, w.size(1) - 1}),
            "the convolution's window must be [B, D, K - 1] of x's type, its weights float32, all contiguous and on one device");
    Tensor z = fresh(x, {B, L, D}), next = fresh(state, state.sizes());
    kla_b200_conv_seq_args c{};
    c.B = B; c.L = L; c.D = D; c.K = w.size(1); c.dtype = dt(x.scalar_type()); c.activation = act;
    c.x = t3(x); c.weight = fp(w); c.bias = fp(bias); c.state = state.data_ptr(); c.state_out = next.data_ptr(); c.z = t3(z);
    check(lib.conv_seq(&c, stream_of(x)));
    return {z, next};
}

// kla_b200_conv_seq_bwd -> dx, dweight, dbias
std::tuple<Tensor, Tensor, OptTensor> conv_seq_bwd(const Tensor &x, const Tensor &dz, const Tensor &w, const OptTensor &bias,
                                                   const Tensor &state, int act) {
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t B = x.size(0), L = x.size(1), D = x.size(2), K = w.size(1);
    Tensor dx = fresh(x, {B, L, D});
    Tensor sums = at::zeros({bias ? D * (K + 1) : D * K}, x.options().dtype(at::kFloat));  // dweight, then dbias
    Tensor dw = sums.narrow(0, 0, D * K).view({D, K});
    OptTensor db;
    if (bias) db = sums.narrow(0, D * K, D);
    kla_b200_conv_seq_bwd_args c{};
    c.B = B; c.L = L; c.D = D; c.K = K; c.dtype = dt(x.scalar_type()); c.activation = act;
    c.x = t3(x); c.dz = t3(dz); c.weight = fp(w); c.bias = fp(bias); c.state = state.data_ptr(); c.dx = t3(dx);
    c.dweight = fp(dw); c.dbias = fp(db);
    check(lib.conv_seq_bwd(&c, stream_of(x)));
    return {dx, dw, db};
}

// One of the four raw scans over [B, L, M, S] coefficients.
void rawscan(int which, const std::vector<Tensor> &ins, const std::vector<Tensor> &outs, const OptTensor &state0, const OptTensor &dstate0) {
    const Tensor &x = ins[0];
    const c10::cuda::CUDAGuard guard(x.device());
    kla_b200_rawscan_args r{};
    r.B = x.size(0); r.L = x.size(1); r.N = x.size(2) * x.size(3);
    for (size_t i = 0; i < ins.size(); ++i) r.in[i] = fp(ins[i]);
    for (size_t i = 0; i < outs.size(); ++i) r.out[i] = fp(outs[i]);
    r.state0 = fp(state0); r.dstate0 = fp(dstate0);
    check(lib.rawscan[which](&r, stream_of(x)));
}

// --------------------------------------------------------------------------------------------------- decode steps

bool wants_grad(std::initializer_list<const Tensor *> ts) {
    if (!c10::GradMode::is_enabled()) return false;
    for (const Tensor *t : ts)
        if (t->requires_grad()) return true;
    return false;
}

// kla_b200_step -> (y, y_var, lam, eta), or None when the arguments need the wrapper's general path.
py::object step(const Tensor &v, const Tensor &lv, const Tensor &k, const Tensor &q, const Tensor &a, const Tensor &p, const Tensor &lam,
                const Tensor &eta, bool prior, bool inplace) {
    if (!v.is_cuda() || v.dim() != 2 || k.dim() != 2 || a.dim() != 2 || lam.dim() != 3) return py::none();
    const auto T = v.scalar_type();
    const int64_t B = v.size(0), M = v.size(1), S = k.size(1);
    if ((T != at::kFloat && T != at::kBFloat16) || lv.scalar_type() != T || k.scalar_type() != T || q.scalar_type() != T) return py::none();
    if (S > KLA_B200_MAX_DSTATE || lv.sizes() != v.sizes() || q.sizes() != k.sizes() || k.size(0) != B || a.size(0) != M || a.size(1) != S ||
        p.sizes() != a.sizes() || lam.size(0) != B || lam.size(1) != M || lam.size(2) != S || eta.sizes() != lam.sizes())
        return py::none();
    for (const Tensor *t : {&a, &p, &lam, &eta})
        if (t->scalar_type() != at::kFloat || !t->is_contiguous()) return py::none();
    for (const Tensor *t : {&lv, &k, &q, &a, &p, &lam, &eta})
        if (t->device() != v.device()) return py::none();
    if (!rows_ok(v) || !rows_ok(lv) || !rows_ok(k) || !rows_ok(q) || !sm100(v.device())) return py::none();
    if (wants_grad({&v, &lv, &k, &q, &a, &p, &lam, &eta})) return py::none();
    const c10::cuda::CUDAGuard guard(v.device());
    Tensor y = f32(v, {B, M}), yv = f32(v, {B, M});
    Tensor lo = inplace ? lam : f32(lam, lam.sizes()), eo = inplace ? eta : f32(eta, eta.sizes());
    kla_b200_step_args s{};
    s.B = B; s.M = M; s.S = S;
    s.in_dtype = dt(T); s.out_dtype = KLA_B200_F32; s.decode_from_prior = prior;
    s.v = v.data_ptr(); s.lambda_v = lv.data_ptr(); s.v_stride_b = v.stride(0); s.lambda_v_stride_b = lv.stride(0);
    s.k = k.data_ptr(); s.q = q.data_ptr(); s.k_stride_b = k.stride(0); s.q_stride_b = q.stride(0);
    s.a = fp(a); s.p = fp(p); s.lam = fp(lam); s.eta = fp(eta);
    s.y = y.data_ptr(); s.y_var = yv.data_ptr(); s.lam_out = fp(lo); s.eta_out = fp(eo);
    check(lib.step(&s, stream_of(v)));
    return py::make_tuple(y, yv, lo, eo);
}

int act_code(const py::object &name) {  // the activation's name in a config, or None
    if (name.is_none()) return KLA_B200_ACT_NONE;
    const std::string s = name.cast<std::string>();
    if (s == "silu") return KLA_B200_ACT_SILU;
    if (s == "gelu") return KLA_B200_ACT_GELU;
    if (s == "relu") return KLA_B200_ACT_RELU;
    throw py::key_error(s);
}

// Whether kla_b200_linear takes the projection: a few bfloat16 rows, nothing to differentiate, vectors aligned; with a norm
// the normalised rows must fit shared memory. The kernel is given pointers, so whatever does not agree in shape or device
// is left to the tensor operations, which raise their own errors.
bool few_rows(const Tensor &x, const Tensor &w, const OptTensor &bias, const OptTensor &norm_w) {
    if (x.dim() != 2 || w.dim() != 2 || !x.is_cuda()) return false;
    const int64_t N = w.size(0), K = w.size(1);
    auto fits = [K](int64_t rows) {  // KLA_B200_LINEAR_SMEM
        int64_t n = 8;
        while (n < rows) n *= 2;
        return n * (K + 8) * 2 + 1024 * (n + 2) <= KLA_B200_LINEAR_SMEM;
    };
    auto plain = [&x](const Tensor &t) { return t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.device() == x.device(); };
    auto vector = [&plain](const OptTensor &t, int64_t n) { return !t || (plain(*t) && t->dim() == 1 && t->size(0) == n); };
    return x.scalar_type() == at::kBFloat16 && x.size(0) >= 1 && x.size(0) <= KLA_B200_LINEAR_MAX_ROWS && x.size(1) == K && K >= 8 &&
           x.stride(1) == 1 && x.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0 && K % 8 == 0 && plain(w) &&
           reinterpret_cast<uintptr_t>(w.data_ptr()) % 16 == 0 && vector(bias, N) && vector(norm_w, K) &&
           (!norm_w || reinterpret_cast<uintptr_t>(norm_w->data_ptr()) % 16 == 0) && fits(x.size(0)) &&
           !wants_grad({&x, &w, bias ? &*bias : &x, norm_w ? &*norm_w : &x}) && sm100(x.device());
}

// Whether a projection that few_rows() takes is faster so than as the library's GEMM with the norm, gate and sum as kernels
// of their own. Up to 16 rows always. Beyond, a CTA brings in (and normalises) four groups of eight rows and keeps half as
// much of W in flight; the library's kernels win as rows x N x K grows. Measured in a CUDA graph, W from HBM, us, kernel
// against library (plain; gate and up with norm and the projection behind; norm with the convolution's step):
//    51 M  24 rows 2080 x 1024 3.4 / 4.3                    75 M  24 rows 4096 x 768 14.8 / 15.8
//    68 M  32 rows 2080 x 1024 3.5 / 4.3                    75 M  32 rows 3072 x 768 9.2 / 8.9
//    67 M  32 rows 1024 x 2048 5.3 / 6.0                    95 M  17 rows 5440 x 1024 23.2 / 18.9
//    81 M  17 rows 3104 x 1536 6.5 / 5.4                   100 M  24 rows 4096 x 1024 10.8 / 9.9
//    89 M  32 rows 1024 x 2720 9.0 / 8.2                   101 M  32 rows 4096 x 768 16.3 / 15.9
//   144 M  17 rows 4128 x 2048 7.6 / 6.4                   134 M  32 rows 4096 x 1024 12.5 / 9.9
bool kernel_pays(int64_t rows, int64_t N, int64_t K) { return rows <= 16 || rows * N * K <= 80'000'000; }
// Rows up to which a token can be one kernel. (Two groups of eight rows, as the kernel was tried: 12 layers d_model 768 16 rows
// 377 us against 371 of the separate kernels.)
constexpr int64_t kTokenRows = KLA_B200_TOKEN_MAX_ROWS;
// Whether that is the faster way for a block, issued from a graph: time of the separate kernels over that of the one, M = 2 d_model,
// swiglu of 8/3 d_model (without an MLP), W from HBM; d_model 128 to 4096, 8 to 128 states, 1, 2, 4, 6 and 8 rows.
// * The filter's units (32 / lanes channels of a row) are dealt one to a warp, and a second round of them costs more from state to
//   state. One round: 1.05 to 1.25 from two rows on, at all sizes; two rounds or more: 16 states 1.02 to 1.23 (0.98 to 1.25), 32 states
//   1.00 to 1.06 up to d_model 1536, 1.00 at 2048 and 8 rows (0.95), 64 states 0.93 to 1.06, 128 states 0.85 to 1.08.
// * One row: up to d_model 384 1.06 to 1.15; beyond, with 32768 states a row or fewer, 1.02 to 1.14 up to d_model 768, 0.98 at 1024
//   (1.07), with more 0.90 to 1.01; d_model 1280 and 1536 0.95 and 1.01 with any; from 2048 on 1.06.
// * Wide projections are slow as kernels of their own: d_model 2560 with its MLP and 3072 1.05 to 1.40 up to 4 M states in all, 0.95
//   to 1.06 with more. Past 6144 channels x leaves W two stages of the ring: d_model 4096 0.81 to 1.00.
// What the rule takes gains 0.97 to 1.40 with an MLP; without one the same but for three points of few and full CTAs of filter units (32
// states d_model 384 and 640 2 rows, 64 states 384 1 row: 0.87 to 0.94).
bool token_pays(int64_t rows, int64_t M, int64_t S, int64_t widest, int64_t sms) {
    if (M > 6144) return false;
    if (widest >= 12288) return rows * M * S <= 4'000'000;
    if (rows == 1 && M > 768 && (M <= 2048 ? M * S > 32768 : M < 4096)) return false;
    int64_t lanes = 1;
    while (4 * lanes < S) lanes *= 2;
    const int64_t channels = 32 / lanes, units = rows * ((M + channels - 1) / channels);
    return units <= 16 * sms || (S <= 32 && rows * M * S <= 800'000);
}
// A lone layer's token is one kernel only where it is issued call by call, four launches costing the host 21 us whatever the
// sizes, and where the kernel takes less than that. us, one kernel / separate ones, eager: 8 rows d_model 256 14.4 / 20.6, 768
// 17.9 / 20.2, 1024 18.7 / 20.7, 2048 40.8 / 39.6; with 32 states 768 21.0 / 21.9, 1024 22.6 / 20.7. Captured, where the kernel's
// working memory is cleared with every replay, the separate ones win: 8 rows d_model 256 16.4 / 14.3, 1024 20.5 / 19.8.
bool few_weights(int64_t d, int64_t M, int64_t S) { return 3 * M * d + 2 * M * (M + S) <= 16'000'000; }
bool lone_token_pays(int64_t B, int64_t d, int64_t M, int64_t S) {
    return few_weights(d, M, S) && B * M * S <= 400'000 &&
           c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None;
}
// Who runs a projection that few_rows() takes: whoever is faster, or what the caller says.
enum class By { size, kernel, library };

struct Extra {  // what kla_b200_linear does besides the projection
    const OptTensor &norm_w;
    double norm_eps = 0.0;
    OptTensor residual;
    bool swiglu = false;
    kla_b200_linear_args conv{};  // its conv_* fields
};

// weights_ready: see kla_b200_linear_args
Tensor linear_rows(const Tensor &x, const Tensor &w, const OptTensor &bias, const Extra &e, bool weights_ready) {
    Tensor out = fresh(x, {x.size(0), e.swiglu ? w.size(0) / 2 : w.size(0)});
    kla_b200_linear_args l = e.conv;
    l.B = x.size(0); l.N = w.size(0); l.K = w.size(1);
    l.x = x.data_ptr(); l.x_stride_b = x.stride(0);
    l.weight = w.data_ptr(); l.bias = bias ? bias->data_ptr() : nullptr;
    l.out = out.data_ptr(); l.out_stride_b = out.stride(0);
    l.norm_weight = e.norm_w ? e.norm_w->data_ptr() : nullptr; l.norm_eps = (float)e.norm_eps;
    l.swiglu = e.swiglu;
    l.weights_ready = weights_ready;
    if (e.residual) { l.residual = e.residual->data_ptr(); l.residual_stride_b = e.residual->stride(0); }
    check(lib.linear(&l, stream_of(x)));
    return out;
}

Tensor rms_norm(const Tensor &x, const Tensor &w, double eps) {  // RMSNorm, src/kla/layers/common.py:45-55
    const Tensor xf = x.to(at::kFloat);
    return (xf * at::rsqrt(xf.pow(2).mean(-1, true) + eps) * w.to(at::kFloat)).to(x.scalar_type());
}

bool vec_rows(const Tensor &t) {  // rows, at least one, that 16-byte accesses can walk
    return t.is_cuda() && t.dim() >= 1 && t.numel() > 0 && t.is_contiguous() && (t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kFloat) && t.size(-1) % 8 == 0 &&
           reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
}

// x + delta (x itself without delta) and its RMSNorm
std::tuple<Tensor, Tensor> add_norm(const Tensor &x, const OptTensor &delta, const Tensor &w, double eps) {
    const c10::cuda::CUDAGuard guard(x.device());
    if (!vec_rows(x) || !vec_rows(w) || w.dim() != 1 || w.size(0) != x.size(-1) || w.device() != x.device() ||
        (delta && (!vec_rows(*delta) || delta->scalar_type() != x.scalar_type() || delta->sizes() != x.sizes() || delta->device() != x.device())) ||
        wants_grad({&x, &w, delta ? &*delta : &x}) || !sm100(x.device())) {
        const Tensor sum = delta ? x + *delta : x;
        return {sum, rms_norm(sum, w, eps)};
    }
    Tensor sum = delta ? fresh(x, x.sizes()) : x, out = fresh(x, x.sizes());
    check(lib.add_norm(x.numel() / x.size(-1), x.size(-1), dt(x.scalar_type()), dt(w.scalar_type()), x.data_ptr(),
                       delta ? delta->data_ptr() : nullptr, w.data_ptr(), (float)eps, sum.data_ptr(), out.data_ptr(), stream_of(x)));
    return {sum, out};
}

// silu(gate) * up of [..., 2 H] rows
Tensor swiglu(const Tensor &gu) {
    const c10::cuda::CUDAGuard guard(gu.device());
    if (!vec_rows(gu) || gu.size(-1) % 16 || wants_grad({&gu}) || !sm100(gu.device())) {
        const auto halves = gu.chunk(2, -1);
        return at::silu(halves[0]) * halves[1];
    }
    auto sizes = gu.sizes().vec();
    sizes.back() /= 2;
    Tensor out = fresh(gu, sizes);
    check(lib.swiglu(gu.numel() / gu.size(-1), sizes.back(), dt(gu.scalar_type()), gu.data_ptr(), out.data_ptr(), stream_of(gu)));
    return out;
}

// k, q [B, L, S] l2-normalised over S, then clamped to [-clip, clip] when clip > 0
std::tuple<Tensor, Tensor> qk_norm(const Tensor &k, const Tensor &q, double clip) {
    const c10::cuda::CUDAGuard guard(k.device());
    const auto T = k.scalar_type();
    if (!k.is_cuda() || (T != at::kFloat && T != at::kBFloat16) || q.scalar_type() != T || k.dim() != 3 || q.sizes() != k.sizes() ||
        !rows_ok(k) || !rows_ok(q) || k.size(2) > KLA_B200_MAX_DSTATE || !sm100(k.device())) {
        auto one = [clip](const Tensor &x) {
            const Tensor y = x / x.norm(2, -1, true).clamp_min(1e-12);
            return clip > 0.0 ? y.clamp(-clip, clip) : y;
        };
        return {one(k), one(q)};
    }
    Tensor ko = fresh(k, k.sizes()), qo = fresh(q, q.sizes());
    check(lib.qk_norm(k.size(0), k.size(1), k.size(2), dt(T), t3(k), t3(q), (float)clip, ko.data_ptr(), qo.data_ptr(), stream_of(k)));
    return {ko, qo};
}

// out[...] (int64) = argmax of x[..., n] over its last dimension; returns out
Tensor argmax(const Tensor &x, Tensor out) {
    const c10::cuda::CUDAGuard guard(x.device());
    const auto T = x.scalar_type();
    if (x.dim() != 2 || x.size(1) < 1 || x.stride(1) != 1 || !x.is_cuda() || (T != at::kFloat && T != at::kBFloat16) || !sm100(x.device()))
        return out.copy_(x.argmax(-1));
    check(lib.argmax(x.size(0), x.size(1), dt(T), x.data_ptr(), x.stride(0), out.data_ptr<int64_t>(), stream_of(x)));
    return out;
}

// A language model's head (a norm in front, no sum behind): from how many outputs on the library's GEMM and the
// norm as a launch of its own are the better read of W. Measured as above, W from HBM, us, kernel / library at one and eight
// rows: K=128 N=4096 2.7 3.9 / 4.1 4.2, N=8192 4.1 5.3 / 4.4 4.8; K=256 N=8192 4.5 5.6 / 5.5 5.7, N=16384 7.9 9.1 / 6.1 6.3;
// K=512 N=8192 4.8 6.1 / 6.7 6.8, N=16384 8.4 9.8 / 7.8 7.9; K=768 N=16384 8.7 10.3 / 9.6 9.7, N=32000 14.6 16.0 / 13.7 13.9;
// K=1024 N=16384 9.4 10.8 / 11.4 11.6, N=50304 23.8 25.5 / 25.7 26.3. At 32 rows the library wins from 4096 outputs on at
// every K (K=256 7.6 / 5.3, K=1024 12.5 / 8.3).
int64_t widest_head(int64_t rows, int64_t K) { return rows <= 16 ? 12 * K + 4096 : 2048; }

// From so many outputs on any other projection is the library's too, at eight rows: 8192 x 1024 7.3 / 5.7, 8224 x 4096
// 15.4 / 13.5, 16384 x 2048 15.0 / 13.6; below, 4128 x 2048 7.0 / 8.0, 4096 x 8192 21.4 / 20.9.
constexpr int64_t kWidePlain = 8192;

// norm (when norm_w is given), projection, residual sum (when given)
Tensor project(const Tensor &x, const Tensor &w, const OptTensor &bias, const OptTensor &norm_w, double eps, const OptTensor &residual,
               bool weights_ready = true, By by = By::size) {
    const c10::cuda::CUDAGuard guard(x.device());
    auto sums = [&] {  // the residual is one the kernel can add
        return !residual || (residual->scalar_type() == at::kBFloat16 && residual->dim() == 2 && residual->size(0) == x.size(0) &&
                             residual->size(1) == w.size(0) && residual->stride(1) == 1 && residual->device() == x.device() &&
                             !wants_grad({&*residual}));
    };
    const bool head = norm_w && !residual;
    auto pays = [&] {
        const int64_t rows = x.size(0), N = w.size(0), K = w.size(1);
        return head ? N <= widest_head(rows, K) : N < kWidePlain && kernel_pays(rows, N, K);
    };
    if (by != By::library && few_rows(x, w, bias, norm_w) && (by == By::kernel || pays()) && sums())
        return linear_rows(x, w, bias, Extra{norm_w, eps, residual}, weights_ready);
    const Tensor out = at::linear(norm_w ? std::get<1>(add_norm(x, {}, *norm_w, eps)) : x, w, bias);
    return residual ? *residual + out : out;
}

struct Weights {  // a layer's weights by name; what a dict does not hold is absent
    const py::dict &d;
    Tensor at(const char *name) const { return d[name].cast<Tensor>(); }
    OptTensor get(const char *name) const {
        const PyObject *o = PyDict_GetItemString(d.ptr(), name);
        return o ? OptTensor(py::handle(const_cast<PyObject *>(o)).cast<Tensor>()) : OptTensor();
    }
    Tensor linear(const Tensor &x, const char *w, const char *b, bool weights_ready, By by) const {
        return project(x, at(w), get(b), {}, 0.0, {}, weights_ready, by);
    }
};

// x + mlp(norm(x)) of one token (src/kla/layers/common.py:99-122): w12, w3 of a swiglu MLP
Tensor swiglu_step(const Tensor &x, const Tensor &norm_w_, double eps, const Tensor &w12, const OptTensor &b12, const Tensor &w3,
                   const OptTensor &b3) {
    const c10::cuda::CUDAGuard guard(x.device());
    const OptTensor norm_w = norm_w_;
    Tensor h;
    if (few_rows(x, w12, b12, norm_w) && w12.size(0) % 2 == 0 && kernel_pays(x.size(0), w12.size(0), w12.size(1))) {
        Extra e{norm_w, eps};
        e.swiglu = true;
        h = linear_rows(x, w12, b12, e, true);
    } else {
        h = swiglu(at::linear(std::get<1>(add_norm(x, {}, norm_w_, eps)), w12, b12));
    }
    return project(h, w3, b3, {}, 0.0, x);
}

// ------------------------------------------------------------------------------------------ a token as one kernel

py::object entry(const py::dict &d, const char *name) {
    PyObject *o = PyDict_GetItemString(d.ptr(), name);
    if (o == nullptr) throw py::key_error(name);
    return py::reinterpret_borrow<py::object>(o);
}

// A layer as ModelDecoder and LayerDecoder hand it over: weights and config by name, what was made of them, its state.
struct LayerArgs {
    const py::dict &w, &cfg;
    const OptTensor &conv_state;
    const Tensor &lam, &eta, &a_bar, &p_bar;
    const OptTensor &skip, &conv_w, &conv_b;
    int64_t w_value, w_var;
};

// Whether kla_b200_token takes the layer for tokens like x; fills l if so. Checks what the kernels are given pointers for, as
// layer_step and few_rows do for the separate ones: whatever does not fit is theirs, with their errors.
bool token_layer(const Tensor &x, const LayerArgs &a, const OptTensor &norm_w, kla_b200_token_layer &l) {
    if (a.a_bar.dim() != 2 || a.w.contains("value_expand.weight") || a.w.contains("var_expand.weight")) return false;
    const auto dev = x.device();
    const int64_t B = x.size(0), d = x.size(1), M = a.a_bar.size(0), S = a.a_bar.size(1);
    const Weights w{a.w};
    const bool gated = entry(a.cfg, "use_gating").cast<bool>();
    if ((a.w_value != 0 && a.w_value != M) || a.w_var != M || M < 8 || M % 8 || S < 1 || S > KLA_B200_MAX_DSTATE) return false;
    if (!is(a.lam, dev, at::kFloat, {B, M, S}) || !is(a.eta, dev, at::kFloat, {B, M, S}) || !is(a.a_bar, dev, at::kFloat, {M, S}) ||
        !is(a.p_bar, dev, at::kFloat, {M, S}))
        return false;
    if (a.skip && !is(*a.skip, dev, at::kFloat, {a.skip->numel() == 1 ? 1 : M})) return false;
    if (a.conv_w) {
        if (a.conv_w->dim() != 2 || a.conv_w->size(1) < 1 || a.conv_w->size(1) > KLA_B200_MAX_CONV_TAPS ||
            !is(*a.conv_w, dev, at::kFloat, {M, a.conv_w->size(1)}) || (a.conv_b && !is(*a.conv_b, dev, at::kFloat, {M})))
            return false;
        if (a.conv_state ? !is(*a.conv_state, dev, at::kBFloat16, {B, M, a.conv_w->size(1) - 1}) : a.conv_w->size(1) != 1) return false;
    }
    auto matrix = [&](const char *name, const char *bias_name, int64_t N, int64_t K, const void *&p, const void *&bias) {
        const OptTensor t = w.get(name), b = w.get(bias_name);
        auto plain = [&](const Tensor &u) { return u.scalar_type() == at::kBFloat16 && u.device() == dev && u.is_contiguous(); };
        if (!t || !plain(*t) || t->dim() != 2 || t->size(0) != N || t->size(1) != K || reinterpret_cast<uintptr_t>(t->data_ptr()) % 16) return false;
        if (b && (!plain(*b) || b->dim() != 1 || b->size(0) != N)) return false;
        if (wants_grad({&*t, b ? &*b : &*t})) return false;
        p = t->data_ptr();
        bias = b ? b->data_ptr() : nullptr;
        return true;
    };
    if (!matrix("in_proj.weight", "in_proj.bias", gated ? 2 * M : M, d, l.in_weight, l.in_bias) ||
        !matrix("sensor_proj.weight", "sensor_proj.bias", a.w_value + a.w_var + 2 * S, M, l.sensor_weight, l.sensor_bias) ||
        !matrix("out_proj.weight", "out_proj.bias", d, M, l.out_weight, l.out_bias))
        return false;
    if (norm_w) {
        if (!few_rows(x, w.at("in_proj.weight"), {}, norm_w)) return false;
        l.norm_weight = norm_w->data_ptr();
    }
    if (a.conv_w) {
        l.conv_weight = fp(*a.conv_w); l.conv_bias = fp(a.conv_b); l.conv_taps = a.conv_w->size(1);
        l.conv_state = a.conv_state ? a.conv_state->data_ptr() : nullptr;
        l.conv_activation = act_code(entry(a.cfg, "conv_activation"));
    }
    const py::object vmax = entry(a.cfg, "obs_var_max"), clip = entry(a.cfg, "clip_value");
    l.a = fp(a.a_bar); l.p = fp(a.p_bar); l.lambda_skip = fp(a.skip); l.lambda_skip_len = a.skip ? (int32_t)a.skip->numel() : 0;
    l.lam = fp(a.lam); l.eta = fp(a.eta);
    l.M = M; l.S = S; l.gated = gated; l.w_value = (int32_t)a.w_value;
    l.gate_activation = gated ? act_code(entry(a.cfg, "gating_activation")) : KLA_B200_ACT_NONE;
    l.qk_norm = entry(a.cfg, "qk_norm").cast<bool>(); l.decode_from_prior = entry(a.cfg, "decode_from_prior").cast<bool>();
    l.obs_var_min = entry(a.cfg, "obs_var_min").cast<float>();
    l.obs_var_max = vmax.is_none() ? 0.0f : vmax.cast<float>();
    l.clip_value = clip.is_none() ? 0.0f : clip.cast<float>();
    return true;
}

// What a token's working memory is good for: launches of one kind.
using TokenKind = std::vector<int64_t>;
TokenKind token_kind(const kla_b200_token_args &t) {
    TokenKind k{t.B, t.d, t.mlp};
    for (int64_t i = 0; i < t.layers; ++i) {
        const kla_b200_token_layer &l = t.layer[i];
        k.insert(k.end(), {l.M, l.S, l.hidden, l.gated, l.w_value});
    }
    return k;
}

// Zeroed working memory for launches of a kind. Launches of one stream follow one another and share it, those of another
// stream have their own: kept by stream (its id is never given to another one) and kind, the last kMost of up to kLargest
// bytes. While a graph is captured it belongs to the graph, whose replays follow one another, and is cleared at its beginning.
Tensor token_work(const Tensor &like, const kla_b200_token_args &t, int64_t bytes) {
    constexpr size_t kMost = 32;
    constexpr int64_t kLargest = 4 << 20;
    struct Kept {
        int device;
        unsigned long long stream;
        TokenKind kind;
        Tensor work;
    };
    // under the interpreter's lock; never destroyed: at exit the CUDA context goes first
    static auto &kept = *new std::vector<Kept>();
    const int device = like.device().index();
    unsigned long long id = 0;
    auto zeros = [&] { return at::zeros({bytes}, like.options().dtype(at::kByte).requires_grad(false)); };
    if (bytes > kLargest || c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None ||
        cudaStreamGetId(at::cuda::getCurrentCUDAStream(device).stream(), &id) != cudaSuccess)
        return zeros();
    TokenKind kind = token_kind(t);
    for (const Kept &k : kept)
        if (k.device == device && k.stream == id && k.kind == kind) return k.work;
    if (kept.size() >= kMost) kept.erase(kept.begin());  // back to the allocator, in the order of the stream that used it
    kept.push_back(Kept{device, id, std::move(kind), zeros()});
    return kept.back().work;
}

// Runs the layers filled in by token_layer -> [B, d], or nothing where a projection's x does not fit the kernel. works: zeroed
// working memory of the caller's, one per KLA_B200_TOKEN_MAX_LAYERS layers; empty: filled with new ones, for the caller to keep.
OptTensor run_token(const Tensor &x, const std::vector<kla_b200_token_layer> &layers, bool mlp, double eps, const OptTensor &y_var,
                    std::optional<py::list> works) {
    std::vector<kla_b200_token_args> runs;
    std::vector<int64_t> bytes;
    for (size_t first = 0; first < layers.size(); first += KLA_B200_TOKEN_MAX_LAYERS) {
        kla_b200_token_args t{};
        t.B = x.size(0); t.d = x.size(1); t.layers = (int64_t)std::min(layers.size() - first, (size_t)KLA_B200_TOKEN_MAX_LAYERS);
        t.mlp = mlp; t.norm_eps = (float)eps;
        t.layer = layers.data() + first;
        bytes.push_back((int64_t)lib.token_work_bytes(&t));
        if (bytes.back() == 0) return {};
        runs.push_back(t);
    }
    Tensor in = x;
    for (size_t i = 0; i < runs.size(); ++i) {
        kla_b200_token_args &t = runs[i];
        if (works && works->size() <= i) works->append(at::zeros({bytes[i]}, x.options().dtype(at::kByte).requires_grad(false)));
        const Tensor work = works ? (*works)[i].cast<Tensor>() : token_work(x, t, bytes[i]);
        require(work.device() == x.device() && work.nbytes() >= (size_t)bytes[i], "a token's working memory belongs to another kind of token");
        Tensor out = fresh(x, {t.B, t.d});
        t.x = in.data_ptr(); t.x_stride_b = in.stride(0);
        t.out = out.data_ptr(); t.y_var = y_var ? y_var->data_ptr() : nullptr;
        t.work = work.data_ptr();
        check(lib.token(&t, stream_of(x)));
        in = out;
    }
    return in;
}

// A row count, type and layout of x that kla_b200_token takes.
bool token_rows(const Tensor &x, int64_t most) {
    return x.is_cuda() && x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.size(0) >= 1 && x.size(0) <= most && x.size(1) >= 8 &&
           x.size(1) % 8 == 0 && x.stride(1) == 1 && x.stride(0) % 8 == 0 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0 &&
           !wants_grad({&x}) && sm100(x.device());
}

// One token through all blocks of a model, or None where a block or the rows are not ones kla_b200_token takes or is the faster way for. blocks: per
// block (weights, config, conv window, lam, eta, a_bar, p_bar, skip, conv weights, conv bias, w_value, w_var, norm weight) and,
// with a swiglu MLP behind the mixer, (norm weight, w12, bias, w3, bias).
using BlockArgs = std::tuple<py::dict, py::dict, OptTensor, Tensor, Tensor, Tensor, Tensor, OptTensor, OptTensor, OptTensor, int64_t, int64_t, Tensor>;
using MlpArgs = std::tuple<Tensor, Tensor, OptTensor, Tensor, OptTensor>;
py::object model_token(const Tensor &x, const std::vector<BlockArgs> &blocks, const std::vector<MlpArgs> &mlps, double eps, std::optional<py::list> works) {
    if (!token_rows(x, kTokenRows) || blocks.empty() || (!mlps.empty() && mlps.size() != blocks.size())) return py::none();
    const c10::cuda::CUDAGuard guard(x.device());
    std::vector<kla_b200_token_layer> layers(blocks.size());
    const int64_t rows = x.size(0), d = x.size(1), sms = at::cuda::getDeviceProperties(x.device().index())->multiProcessorCount;
    // Issued call by call, a block's separate kernels cost the host 30 us, which is more than they take up to the sizes of a lone
    // layer's rule.
    const bool replayed = works || c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
    for (size_t i = 0; i < blocks.size(); ++i) {
        const auto &[w, cfg, conv_state, lam, eta, a_bar, p_bar, skip, conv_w, conv_b, w_value, w_var, norm_w] = blocks[i];
        if (!token_layer(x, LayerArgs{w, cfg, conv_state, lam, eta, a_bar, p_bar, skip, conv_w, conv_b, w_value, w_var}, norm_w, layers[i])) return py::none();
        const int64_t M = layers[i].M, S = layers[i].S, hidden_out = mlps.empty() || std::get<1>(mlps[i]).dim() != 2 ? 0 : std::get<1>(mlps[i]).size(0);
        if ((replayed || !few_weights(d, M, S)) && !token_pays(rows, M, S, std::max((layers[i].gated ? 2 : 1) * M, hidden_out), sms)) return py::none();
        if (mlps.empty()) continue;
        const auto &[mlp_norm, w12, b12, w3, b3] = mlps[i];
        const int64_t hidden = w12.dim() == 2 ? w12.size(0) / 2 : 0;
        if (!few_rows(x, w12, b12, mlp_norm) || w12.size(0) != 2 * hidden || hidden < 8 || hidden % 8) return py::none();
        if (w3.dim() != 2 || w3.size(0) != x.size(1) || w3.size(1) != hidden || w3.scalar_type() != at::kBFloat16 || !w3.is_contiguous() || w3.device() != x.device() ||
            reinterpret_cast<uintptr_t>(w3.data_ptr()) % 16 || wants_grad({&w3}) ||
            (b3 && (b3->scalar_type() != at::kBFloat16 || !b3->is_contiguous() || b3->dim() != 1 || b3->size(0) != w3.size(0) || b3->device() != x.device() || wants_grad({&*b3}))))
            return py::none();
        layers[i].mlp_norm_weight = mlp_norm.data_ptr(); layers[i].w12 = w12.data_ptr(); layers[i].b12 = b12 ? b12->data_ptr() : nullptr;
        layers[i].w3 = w3.data_ptr(); layers[i].b3 = b3 ? b3->data_ptr() : nullptr; layers[i].hidden = hidden;
    }
    return py::cast(run_token(x, layers, !mlps.empty(), eps, {}, works));
}

// One token of a layer (LayerDecoder.step), with the block's norm before it and its residual sum after it when norm_w is given
// (ModelDecoder): three projections, the convolution's step and the fused filter step, or one kernel where that pays and may take
// the whole GPU. conv_state
// (absent without a convolution), lam and eta are updated in place. Returns the layer's output and the gated variance, which
// a config that returns variances projects as well.
std::tuple<Tensor, Tensor> layer_step(const py::dict &w_, const py::dict &cfg, const Tensor &x, const OptTensor &conv_state,
                                      const Tensor &lam, const Tensor &eta, const Tensor &a_bar, const Tensor &p_bar,
                                      const OptTensor &skip, const OptTensor &conv_w, const OptTensor &conv_b, int64_t w_value,
                                      int64_t w_var, const OptTensor &norm_w, double norm_eps, bool whole) {
    const c10::cuda::CUDAGuard guard(x.device());
    const Weights w{w_};
    auto get = [&cfg](const char *name) {
        PyObject *o = PyDict_GetItemString(cfg.ptr(), name);
        if (o == nullptr) throw py::key_error(name);
        return py::reinterpret_borrow<py::object>(o);
    };
    void *stream = stream_of(x);
    require_type(x);
    require(x.dim() == 2 && a_bar.dim() == 2, "a token is [B, d_model]");
    const auto dev = x.device();
    const int64_t B = x.size(0), M = a_bar.size(0), S = a_bar.size(1);
    const int32_t type = dt(x.scalar_type());
    const bool gated = get("use_gating").cast<bool>();
    for (const Tensor *t : {&lam, &eta}) require(is(*t, dev, at::kFloat, {B, M, S}), "the filter state must be contiguous float32 [B, M, S] on x's device");
    for (const Tensor *t : {&a_bar, &p_bar}) require(is(*t, dev, at::kFloat, {M, S}), "a_bar and p_bar must be contiguous float32 [M, S] on x's device");
    require(!skip || is(*skip, dev, at::kFloat, {skip->numel() == 1 ? 1 : M}), "the skip weights must be one float32 value or one per channel, on x's device");
    if (conv_w) {
        require(conv_w->dim() == 2 && is(*conv_w, dev, at::kFloat, {M, conv_w->size(1)}) && (!conv_b || is(*conv_b, dev, at::kFloat, {M})),
                "the convolution's weights must be contiguous float32 [M, K] and [M] on x's device");
        require(conv_state ? is(*conv_state, dev, x.scalar_type(), {B, M, conv_w->size(1) - 1}) : conv_w->size(1) == 1,
                "the convolution's window must be contiguous [B, M, K - 1] of x's type on its device");
    }
    const Tensor in_w = w.at("in_proj.weight");
    const OptTensor in_b = w.get("in_proj.bias");
    const Tensor sensor_w = w.at("sensor_proj.weight");
    const bool in_model = norm_w.has_value();  // other kernels of the token, or the embedding's, are in front
    require(in_w.dim() == 2 && in_w.size(0) == (gated ? 2 * M : M), "in_proj must have one output per channel, two with a gate");
    require(sensor_w.dim() == 2 && sensor_w.size(0) == w_value + w_var + 2 * S, "sensor_proj must have one output per sensor signal");
    if (whole && !in_model && token_rows(x, kTokenRows) && lone_token_pays(B, x.size(1), M, S)) {
        std::vector<kla_b200_token_layer> one(1);
        if (token_layer(x, LayerArgs{w_, cfg, conv_state, lam, eta, a_bar, p_bar, skip, conv_w, conv_b, w_value, w_var}, {}, one[0])) {
            const Tensor yv = fresh(x, {B, M});
            if (const OptTensor out = run_token(x, one, false, 0.0, yv, {})) return {*out, yv};
        }
    }
    // A lone layer issued call by call is bound by the host, where the library's calls cost 7 us more each (B=17 d_model 768:
    // 23.0 us a token, 26.5 with one of them); in a graph its three GEMMs win together where the widest does (d_model 768, B=17
    // 21.9 against 19.0, B=32 28.6 and 21.8; d_model 1024, B=32 27.6 and 24.3; but d_model 512, B=32 15.7 and 16.6).
    By by = By::size;
    if (!in_model) {
        by = By::kernel;
        if (!kernel_pays(B, sensor_w.size(0), sensor_w.size(1)) &&
            c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) {
            by = By::library;
            // The eager tokens before the capture did not use the library: it may have to set itself up now, which the other
            // capture modes would not let it.
            const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
            at::cuda::getCurrentCUDABlasHandle();
        }
    }
    // with the kernel the convolution's step rides on the first projection
    const bool fused = by != By::library && few_rows(x, in_w, in_b, norm_w) && (by == By::kernel || kernel_pays(B, in_w.size(0), in_w.size(1)));
    Tensor projected;
    if (fused) {
        Extra e{norm_w, norm_eps};
        if (conv_w) {
            e.conv.conv_D = M; e.conv.conv_taps = conv_w->size(1); e.conv.conv_activation = act_code(get("conv_activation"));
            e.conv.conv_weight = fp(*conv_w); e.conv.conv_bias = fp(conv_b);
            e.conv.conv_state = conv_state ? conv_state->data_ptr() : nullptr;
        }
        projected = linear_rows(x, in_w, in_b, e, in_model);
    } else {
        projected = at::linear(norm_w ? std::get<1>(add_norm(x, {}, *norm_w, norm_eps)) : x, in_w, in_b).to(x.scalar_type());
    }
    // The kernels read x's type; under autocast the projections come in another.
    // z and the gate are halves of the projection, the sensor signals slices of theirs: pointers, not views
    const int64_t esz = x.element_size();
    auto part = [esz](const Tensor &t, int64_t column) { return static_cast<char *>(t.data_ptr()) + column * esz; };
    void *z = projected.data_ptr(), *gate = gated ? part(projected, M) : nullptr;
    const int64_t gate_row = gated ? projected.stride(0) : 0;
    int64_t z_row = projected.stride(0);
    Tensor z_in = gated ? projected.narrow(1, 0, M) : projected;  // what sensor_proj reads
    // What runs in front of a lone layer may write its weights, and may let its successor start before it has (these kernels
    // do): the first kernel of the token reads its weights only after it (B=32 d_model 1024, tokens back to back: 28.9 against
    // 28.2 us).
    bool weights_ready = fused || in_model;
    if (conv_w && !fused) {
        Tensor zc = fresh(x, {B, M});
        kla_b200_conv_step_args c{};
        c.B = B; c.D = M; c.K = conv_w->size(1); c.dtype = type;
        c.activation = act_code(get("conv_activation"));
        c.x = z; c.x_stride_b = z_row; c.weight = fp(*conv_w); c.bias = fp(conv_b);
        c.state = conv_state ? conv_state->data_ptr() : nullptr; c.z = zc.data_ptr();
        check(lib.conv_step(&c, stream));
        z_in = zc;
        z = zc.data_ptr();
        z_row = M;
        weights_ready = true;
    }
    const Tensor sens = project(z_in, sensor_w, w.get("sensor_proj.bias"), {}, 0.0, {}, weights_ready, by).to(x.scalar_type());
    const int64_t row = sens.stride(0);
    // the four sensor signals, raw, as KLALayer._project_sensors splits them (src/kla/layers/kla_layer.py:199-216)
    void *v = z, *ls = part(sens, w_value), *kq = part(sens, w_value + w_var);
    int64_t v_row = z_row, ls_row = row;
    Tensor v_wide, ls_wide;  // low-rank signals, expanded
    if (w_value != 0) {
        v = sens.data_ptr();
        v_row = row;
        if (w_.contains("value_expand.weight")) {
            v_wide = w.linear(sens.narrow(1, 0, w_value), "value_expand.weight", "value_expand.bias", weights_ready, by).to(x.scalar_type());
            v = v_wide.data_ptr();
            v_row = v_wide.stride(0);
        }
        require((v_wide.defined() ? v_wide.size(1) : w_value) == M, "there must be one value per channel");
    }
    if (w_.contains("var_expand.weight")) {
        ls_wide = w.linear(sens.narrow(1, w_value, w_var), "var_expand.weight", "var_expand.bias", weights_ready, by).to(x.scalar_type());
        ls = ls_wide.data_ptr();
        ls_row = ls_wide.stride(0);
    }
    require((ls_wide.defined() ? ls_wide.size(1) : w_var) == M, "there must be one log-variance per channel");
    Tensor y = fresh(x, {B, M}), yv = fresh(x, {B, M});
    const py::object vmax = get("obs_var_max"), clip = get("clip_value");
    kla_b200_step_layer_args s{};
    s.B = B; s.M = M; s.S = S; s.in_dtype = type; s.out_dtype = type;
    s.decode_from_prior = get("decode_from_prior").cast<bool>();
    s.qk_norm = get("qk_norm").cast<bool>();
    s.gate_activation = gated ? act_code(get("gating_activation")) : KLA_B200_ACT_NONE;
    s.lambda_skip_len = skip ? (int32_t)skip->numel() : 0;
    s.obs_var_min = get("obs_var_min").cast<float>();
    s.obs_var_max = vmax.is_none() ? 0.0f : vmax.cast<float>();
    s.clip_value = clip.is_none() ? 0.0f : clip.cast<float>();
    s.v = v; s.log_sigma_v = ls; s.v_stride_b = v_row; s.log_sigma_v_stride_b = ls_row;
    s.k = kq; s.q = static_cast<char *>(kq) + S * esz; s.k_stride_b = row; s.q_stride_b = row;
    s.z = z; s.z_stride_b = z_row;
    s.gate = gate; s.gate_stride_b = gate_row;
    s.lambda_skip = fp(skip); s.a = fp(a_bar); s.p = fp(p_bar); s.lam = fp(lam); s.eta = fp(eta);
    s.y = y.data_ptr(); s.y_var = yv.data_ptr(); s.lam_out = fp(lam); s.eta_out = fp(eta);
    s.weights_ready = weights_ready;
    check(lib.step_layer(&s, stream));
    return {project(y, w.at("out_proj.weight"), w.get("out_proj.bias"), {}, 0.0, norm_w ? OptTensor(x) : OptTensor(), true, by), yv};
}

// What a captured step would read: address, type and layout of each tensor. 220 of them take 18 us, as Python tuples 1000.
py::bytes stamp(const std::vector<OptTensor> &ts) {
    std::vector<int64_t> v;
    v.reserve(ts.size() * 8);
    for (const OptTensor &t : ts) {
        if (!t) {
            v.push_back(-1);
            continue;
        }
        v.insert(v.end(), {(int64_t)reinterpret_cast<uintptr_t>(t->data_ptr()), (int64_t)t->scalar_type(), (int64_t)t->device().index(), t->dim()});
        v.insert(v.end(), t->sizes().begin(), t->sizes().end());
        v.insert(v.end(), t->strides().begin(), t->strides().end());
    }
    return py::bytes(reinterpret_cast<const char *>(v.data()), v.size() * sizeof(int64_t));
}

// Whether the GPU is past a recorded event; while another thread captures a graph as well, which a plain query would end.
bool event_done(uintptr_t event) {
    const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
    if (cudaEventQuery(reinterpret_cast<cudaEvent_t>(event)) != cudaErrorNotReady) return true;
    (void)cudaGetLastError();
    return false;
}

}  // namespace

PYBIND11_MODULE(_kla_host, m) {
    m.doc() = "Launches of the kla_b200 library on torch tensors";
    m.def("bind", &bind);
    m.def("canonical", &canonical);
    m.def("scan_fwd", &scan_fwd);
    m.def("scan_bwd", &scan_bwd);
    m.def("slab_aggregate", &slab_aggregate);
    m.def("scan_fwd_chunked", &scan_fwd_chunked);
    m.def("scan_bwd_chunked", &scan_bwd_chunked);
    m.def("epilogue_bwd", &epilogue_bwd);
    m.def("conv_seq", &conv_seq);
    m.def("conv_seq_bwd", &conv_seq_bwd);
    m.def("rawscan", &rawscan);
    m.def("step", &step);
    m.def("layer_step", &layer_step);
    m.def("model_token", &model_token);
    m.def("token_pays", &token_pays);
    m.def("event_done", &event_done);
    m.def("add_norm", &add_norm);
    m.def("swiglu", &swiglu);
    m.def("argmax", &argmax);
    m.def("qk_norm", &qk_norm);
    // one of several kernels of a token, none of which writes weights
    m.def("project", [](const Tensor &x, const Tensor &w, const OptTensor &bias, const OptTensor &norm_w, double eps, const OptTensor &residual) {
        return project(x, w, bias, norm_w, eps, residual);
    });
    m.def("swiglu_step", &swiglu_step);
    m.def("stamp", &stamp);
}
