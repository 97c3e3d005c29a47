"""The decode projections (norm, convolution step, swiglu and residual folded in) against plain float32 torch."""

import importlib
import os
import subprocess
import sys

import pytest
import torch
import torch.nn.functional as F

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
import kla_b200  # noqa: E402,F401

pytestmark = pytest.mark.gpu
lib = importlib.import_module("kalman-linear-attention_b200._lib")
decode = importlib.import_module("kalman-linear-attention_b200.decode")


def close(got, want):
    assert got.dtype == torch.bfloat16 and got.shape == want.shape
    torch.testing.assert_close(got.float(), want, rtol=1e-2, atol=1e-2 * want.abs().mean().item())


def norm(x, w, eps):
    x = x.float()
    return (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.float()).bfloat16().float()


# rows around the groups of eight, K with a part of a 32-column block, N with a part of a 16-row tile and beyond one pass
@pytest.mark.parametrize("B,N,K", [(1, 1, 8), (7, 33, 40), (8, 64, 256), (9, 130, 264), (17, 48, 1024), (32, 100, 72), (31, 4096, 512),
                                   (3, 8000, 64)])
def test_projection_with_norm_bias_and_residual(B, N, K):
    g = torch.Generator(device="cuda").manual_seed(N)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, b, nw, res = rn(B, K + 8)[:, :K], rn(N, K) * K ** -0.5, rn(N), rn(K), rn(B, N)
    n0 = lib.load().kla_b200_launch_count()
    close(lib.host().project(x, w, None, None, 0.0, None), F.linear(x.float(), w.float()))
    close(lib.host().project(x, w, b, nw, 1e-6, res), F.linear(norm(x, nw, 1e-6), w.float(), b.float()) + res.float())
    assert lib.load().kla_b200_launch_count() - n0 == 2


@pytest.mark.parametrize("B,H,K", [(3, 24, 40), (12, 40, 256), (32, 33, 512)])
def test_gate_and_up_of_rows_taken_as_they_are(B, H, K):
    """The C entry's swiglu without a norm in front, which the wrappers do not use."""
    import ctypes

    g = torch.Generator(device="cuda").manual_seed(H)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, b, out = rn(B, K), rn(2 * H, K) * K ** -0.5, rn(2 * H), torch.empty(B, H, device="cuda", dtype=torch.bfloat16)
    lib.check(lib.load().kla_b200_linear(ctypes.byref(lib.LinearArgs(
        B=B, N=2 * H, K=K, x=x.data_ptr(), x_stride_b=K, weight=w.data_ptr(), bias=b.data_ptr(), out=out.data_ptr(), out_stride_b=H, swiglu=1)),
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    gate, up = F.linear(x.float(), w.float(), b.float()).chunk(2, dim=-1)
    close(out, F.silu(gate) * up)


# both sides of the line between the kernel and the library's GEMM beyond 16 rows (80 M multiply-adds), and of a head's
@pytest.mark.parametrize("B,N,K,launches", [(16, 4128, 2048, 1), (17, 4128, 1136, 1), (17, 4128, 1144, 0), (32, 2496, 1000, 1), (32, 2504, 1000, 0)])
def test_large_projections_beyond_sixteen_rows_go_to_the_library(B, N, K, launches):
    g = torch.Generator(device="cuda").manual_seed(N)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, b = rn(B, K), rn(N, K) * K ** -0.5, rn(N)
    n0 = lib.load().kla_b200_launch_count()
    close(lib.host().project(x, w, b, None, 0.0, None), F.linear(x.float(), w.float(), b.float()))
    assert lib.load().kla_b200_launch_count() - n0 == launches


@pytest.mark.parametrize("B,N,K", [(8, 4864, 64), (8, 4872, 64), (17, 2048, 64), (17, 2056, 64)])
def test_heads_on_both_sides_of_the_line(B, N, K):
    g = torch.Generator(device="cuda").manual_seed(N)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w, nw = rn(B, K), rn(N, K) * K ** -0.5, rn(K)
    close(lib.host().project(x, w, None, nw, 1e-6, None), F.linear(norm(x, nw, 1e-6), w.float()))


@pytest.mark.parametrize("B,H,K", [(2, 24, 40), (8, 2048, 768), (20, 40, 256), (32, 33, 512)])
def test_swiglu_step(B, H, K):
    g = torch.Generator(device="cuda").manual_seed(H)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, nw, w12, w3 = rn(B, K), rn(K), rn(2 * H, K) * K ** -0.5, rn(K, H) * H ** -0.5
    gate, up = F.linear(norm(x, nw, 1e-5), w12.float()).chunk(2, dim=-1)
    close(lib.host().swiglu_step(x, nw, 1e-5, w12, None, w3, None), x.float() + F.linear((F.silu(gate) * up).bfloat16().float(), w3.float()))


@pytest.mark.parametrize("B,d", [(1, 64), (11, 48), (32, 72), (64, 128)])
def test_layer_token_in_bfloat16_follows_float32(B, d):
    """The fused token of a bfloat16 layer against the same layer in float32, whose route is the library's GEMMs and the
    convolution and filter kernels one by one; at 64 rows, the library's GEMMs in both. Rounding to bfloat16 changes a tensor
    by 1.7e-3 of its norm (up to 2^-8 of each value). Between x and the output six tensors are rounded (the projections,
    the gate, the convolution's and the filter's outputs): 4.1e-3 in quadrature, and half as much again for what the gate,
    the activations and the state make of it. The window is rounded once; so is what lam is made of."""
    M, S, K = 2 * d, 16, 4
    g = torch.Generator().manual_seed(B)
    rn = lambda *s: torch.randn(*s, generator=g)
    w = {"in_proj.weight": rn(2 * M, d) * d ** -0.5, "sensor_proj.weight": rn(2 * M + 2 * S, M) * M ** -0.5,
         "out_proj.weight": rn(d, M) * M ** -0.5, "conv.weight": rn(M, 1, K) * 0.5, "conv.bias": rn(M) * 0.1, "delta": rn(M, S) - 4,
         "lambda_log": rn(M, S) * 0.1, "process_noise": torch.full((M, S), 0.01), "lambda_skip": torch.tensor(-1.0)}
    w = {k: v.bfloat16().float() if k.endswith("proj.weight") else v for k, v in w.items()}
    cfg = dict(d_state=S, discretization="ou", zero_process_noise=False, clip_value=None, obs_var_min=1e-4, obs_var_max=None,
               value_rank="full", qk_norm=True, use_conv=True, conv_kernel_size=K, conv_activation="silu", use_gating=True,
               gating_activation="silu", use_lambda_skip=True, return_variance=False, decode_from_prior=False)
    f32 = decode.LayerDecoder(w, cfg).to("cuda")
    b16 = decode.LayerDecoder({k: v.bfloat16() if k.endswith("proj.weight") else v for k, v in w.items()}, cfg).to("cuda")
    sa, sb = f32.init_state(B, "cuda"), b16.init_state(B, "cuda", torch.bfloat16)
    for _ in range(5):
        x = rn(B, d).bfloat16().cuda()
        want, got = f32.step(x.float(), sa), b16.step(x, sb)
    rel = lambda a, b: ((a.float() - b.float()).norm() / b.float().norm()).item()
    assert rel(got, want) < 6.2e-3 and rel(sb[2], sa[2]) < 6.2e-3 and rel(sb[0], sa[0]) < 2.5e-3 and rel(sb[1], sa[1]) < 2.5e-3
    torch.testing.assert_close(got.float(), want, rtol=5e-2, atol=3e-2 * want.abs().mean().item() + 1e-2)
    torch.testing.assert_close(sb[0].float(), sa[0], rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(sb[1], sa[1], rtol=5e-2, atol=5e-2)


def test_a_captured_token_of_a_large_layer_follows_the_eager_one():
    """Between 17 and 32 rows a large layer's projections are the library's while a graph is captured. Both routes round
    the same float32 sums once; a sum that falls on the other side changes a result by 2^-8 of it."""
    B, d, S, K = 24, 768, 16, 4
    M = 2 * d
    g = torch.Generator(device="cuda").manual_seed(0)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    w = {"in_proj.weight": (rn(2 * M, d) * d ** -0.5).bfloat16(), "sensor_proj.weight": (rn(2 * M + 2 * S, M) * M ** -0.5).bfloat16(),
         "out_proj.weight": (rn(d, M) * M ** -0.5).bfloat16(), "conv.weight": rn(M, 1, K) * 0.5, "conv.bias": rn(M) * 0.1,
         "delta": rn(M, S) - 4, "lambda_log": rn(M, S) * 0.1, "process_noise": torch.full((M, S), 0.01, device="cuda"),
         "lambda_skip": torch.tensor(-1.0, device="cuda")}
    cfg = dict(d_state=S, discretization="ou", zero_process_noise=False, clip_value=None, obs_var_min=1e-4, obs_var_max=None,
               value_rank="full", qk_norm=True, use_conv=True, conv_kernel_size=K, conv_activation="silu", use_gating=True,
               gating_activation="silu", use_lambda_skip=True, return_variance=False, decode_from_prior=False)
    dec, x = decode.LayerDecoder(w, cfg), rn(B, d).bfloat16()
    eager, state = dec.init_state(B, "cuda", torch.bfloat16), dec.init_state(B, "cuda", torch.bfloat16)
    launched = []

    def token(st):
        n0 = lib.load().kla_b200_launch_count()
        out = dec.step(x, st)
        launched.append(lib.load().kla_b200_launch_count() - n0)
        return out

    want = token(eager)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = token(state)
    graph.replay()
    torch.cuda.synchronize()
    assert launched == [4, 2]
    for a, b in ((got, want), *zip(state, eager)):
        assert (a.float() - b.float()).norm() <= 2 ** -7 * b.float().norm()


def test_a_large_layer_is_captured_before_the_library_has_run():
    """In a process whose tokens so far were all kernels of this package, the capture itself sets the library up."""
    code = """
import importlib, sys
import torch
sys.path.insert(0, %r)
import kla_b200
B, d, S = 24, 768, 16
M = 2 * d
rn = lambda *s: torch.randn(*s, device="cuda")
w = {"in_proj.weight": (rn(2 * M, d) * d ** -0.5).bfloat16(), "sensor_proj.weight": (rn(2 * M + 2 * S, M) * M ** -0.5).bfloat16(),
     "out_proj.weight": (rn(d, M) * M ** -0.5).bfloat16(), "delta": rn(M, S) - 4, "lambda_log": rn(M, S) * 0.1,
     "process_noise": torch.full((M, S), 0.01, device="cuda")}
cfg = dict(d_state=S, discretization="ou", zero_process_noise=False, clip_value=None, obs_var_min=1e-4, obs_var_max=None,
           value_rank="full", qk_norm=True, use_conv=False, conv_kernel_size=4, conv_activation="silu", use_gating=True,
           gating_activation="silu", use_lambda_skip=False, return_variance=False, decode_from_prior=False)
dec, x = kla_b200.LayerDecoder(w, cfg), rn(B, d).bfloat16()
a, b = dec.init_state(B, "cuda", torch.bfloat16), dec.init_state(B, "cuda", torch.bfloat16)
want = dec.step(x, a)
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    got = dec.step(x, b)
g.replay()
torch.cuda.synchronize()
assert (got.float() - want.float()).norm() <= 2 ** -7 * want.float().norm()
""" % os.path.dirname(HERE)
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]


# a row within the registers, across them, and one that does not divide into vectors
@pytest.mark.parametrize("rows,D", [(1, 8), (5, 768), (33, 1032), (7, 4096), (4, 36)])
@pytest.mark.parametrize("dtype,wtype", [(torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32), (torch.float32, torch.float32)])
def test_residual_sum_norm_and_gate(rows, D, dtype, wtype):
    g = torch.Generator(device="cuda").manual_seed(D)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda")
    x, d, w = rn(2, rows, D).to(dtype), rn(2, rows, D).to(dtype), rn(D).to(wtype)
    tol = dict(rtol=1e-2, atol=1e-2) if dtype == torch.bfloat16 else dict(rtol=2e-6, atol=2e-6)
    for delta in (None, d):
        s, out = lib.host().add_norm(x, delta, w, 1e-6)
        want = x if delta is None else x + d
        assert torch.equal(s, want)
        ref = want.double() * torch.rsqrt(want.double().pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
        torch.testing.assert_close(out.double(), ref, **tol)
    a, b = x.double().chunk(2, dim=-1)
    torch.testing.assert_close(lib.host().swiglu(x).double(), F.silu(a) * b, **tol)


@pytest.mark.parametrize("rows,n", [(1, 1), (3, 7), (8, 50304), (5, 8200), (2, 1023)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_greedy_choice(rows, n, dtype):
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(rows, n, generator=g, device="cuda").to(dtype)  # bfloat16: the largest value is often there twice
    got = lib.host().argmax(x, torch.empty(rows, device="cuda", dtype=torch.long))
    first = (x == x.max(dim=-1, keepdim=True).values).long().argmax(dim=-1)
    assert torch.equal(got, first)
    x[-1, n // 2:] = float("nan")
    assert lib.host().argmax(x, got)[-1] == n // 2


@pytest.mark.parametrize("B,L,S,clip", [(1, 1, 1, 0.0), (2, 5, 16, 0.0), (1, 3, 17, 0.3), (3, 2, 100, 0.05), (1, 4, 128, 0.0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_keys_and_queries_are_normalised_and_clipped(B, L, S, clip, dtype):
    g = torch.Generator(device="cuda").manual_seed(S)
    wide = torch.randn(B, L, 2 * S + 3, generator=g, device="cuda").to(dtype)  # slices of a projection
    k, q = wide[..., 1:1 + S], wide[..., S + 2:2 * S + 2]
    k[0, 0] = 0
    tol = dict(rtol=1e-2, atol=1e-3) if dtype == torch.bfloat16 else dict(rtol=1e-6, atol=1e-7)
    for got, x in zip(lib.host().qk_norm(k, q, clip), (k, q)):
        want = x.double() / x.double().norm(dim=-1, keepdim=True).clamp_min(1e-12)
        assert got.dtype == dtype and got.is_contiguous()
        torch.testing.assert_close(got.double(), want.clamp(-clip, clip) if clip else want, **tol)


@pytest.mark.parametrize("clip", [0.0, 0.3])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_keys_that_are_not_finite_stay_so(clip, dtype):
    x = torch.randn(1, 5, 20, device="cuda").to(dtype)
    x[0, 1, 3], x[0, 2, 19], x[0, 3, 0] = float("nan"), float("inf"), float("-inf")
    want = x.double() / x.double().norm(dim=-1, keepdim=True).clamp_min(1e-12)
    want = want.clamp(-clip, clip) if clip else want
    for got in lib.host().qk_norm(x, x, clip):
        torch.testing.assert_close(got.double(), want, rtol=1e-2, atol=1e-3, equal_nan=True)


def test_shapes_that_do_not_agree_raise_or_broadcast_as_tensor_operations_do():
    """The kernels are given pointers: a row shorter than the weights' is for the tensor operations to refuse."""
    rn = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    host, B, N, K = lib.host(), 4, 48, 64
    w, norm_w, res = rn(N, K), rn(K), rn(B, N)
    for x in (rn(B, K - 8), rn(B, K + 8), rn(B, 8)):
        with pytest.raises(RuntimeError):
            host.project(x, w, None, None, 0.0, None)
        with pytest.raises(RuntimeError):
            host.project(x, w, None, norm_w, 1e-6, None)
        with pytest.raises(RuntimeError):
            host.swiglu_step(x, norm_w, 1e-6, w, None, rn(K, N // 2), None)
    x = rn(B, K)
    for bad in (dict(bias=rn(N - 8)), dict(norm=rn(K // 2)), dict(res=rn(B, N - 8)), dict(res=rn(B - 1, N)), dict(bias=rn(N).cpu()),
                dict(norm=rn(K).cpu())):
        with pytest.raises(RuntimeError):
            host.project(x, w, bad.get("bias"), bad.get("norm"), 1e-6, bad.get("res"))
    with pytest.raises(RuntimeError):  # the MLP's output is narrower than what it is added to
        host.swiglu_step(x, norm_w, 1e-6, w, None, rn(K - 8, N // 2), None)
    for wrong in (rn(K - 8), rn(2 * K)):
        with pytest.raises(RuntimeError):
            host.add_norm(x, None, wrong, 1e-6)
    with pytest.raises(RuntimeError):
        host.add_norm(x, rn(B, K - 8), norm_w, 1e-6)
    # one value for all columns, one row for all rows: broadcast
    one = rn(1)
    close(host.add_norm(x, None, one, 1e-6)[1], norm(x, one, 1e-6))
    close(host.project(x, w, None, None, 0.0, res[:1]), F.linear(x.float(), w.float()) + res[:1].float())
    assert host.add_norm(rn(0, K), None, norm_w, 1e-6)[1].shape == (0, K) and host.swiglu(rn(0, K)).shape == (0, K // 2)
    assert host.add_norm(rn(B, 0), None, rn(0), 1e-6)[1].shape == (B, 0) and host.swiglu(rn(B, 0)).shape == (B, 0)
