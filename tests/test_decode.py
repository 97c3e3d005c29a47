"""Layer decode (conv step + fused sensor/filter/gate step): the B200 kernels against the
reference layer's own token-by-token outputs (tests/golden/decode_*.npz)."""

import glob
import os
import sys

import numpy as np
import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
import kla_b200  # noqa: E402
from conftest import reference_src  # noqa: E402
from importlib import import_module  # noqa: E402

decode = import_module("kalman-linear-attention_b200.decode")
CASES = sorted(os.path.basename(p)[7:-4] for p in glob.glob(os.path.join(HERE, "golden", "decode_*.npz")))
REF_SRC = reference_src()  # the directory holding the reference package `kla`, or "" when there is none here
needs_ref = pytest.mark.skipif(not os.path.isdir(REF_SRC), reason="reference package not present")


def load(name):
    z = dict(np.load(os.path.join(HERE, "golden", f"decode_{name}.npz")))
    weights = {k[2:]: torch.from_numpy(v) for k, v in z.items() if k.startswith("w:")}
    config = {}
    for k, v in z.items():
        if k.startswith("c:"):
            val = v.item()
            config[k[2:]] = None if val == "" else val
    return z, weights, config


def test_cases_present():
    assert CASES == ["bare", "default", "lowrank", "variant"]


@pytest.mark.parametrize("name", CASES)
def test_discretisation_matches_the_layer(name):
    z, weights, config = load(name)
    a_bar, p_bar = decode.discretize(weights, config)
    np.testing.assert_allclose(a_bar.numpy(), z["a_bar"], rtol=1e-6, atol=1e-8)
    np.testing.assert_allclose(p_bar.numpy(), z["p_bar"], rtol=1e-6, atol=1e-10)
    dec = kla_b200.LayerDecoder(weights, config)
    assert (dec.M, dec.S) == z["lam0"].shape[1:]
    assert dec.w_value + dec.w_var + 2 * dec.S == weights["sensor_proj.weight"].shape[0]


def test_cpu_tensors_are_refused():
    _, weights, config = load("default")
    dec = kla_b200.LayerDecoder(weights, config)
    with pytest.raises(NotImplementedError, match="CUDA"):
        dec.step(torch.zeros(2, 32), dec.init_state(2, "cpu"))
    with pytest.raises(ValueError, match="lacks"):
        kla_b200.LayerDecoder(weights, {"d_state": 8})


def tiny_model(d=32, M=64, S=16, layers=1, vocab=24, dtype=torch.float32):
    """A ``ModelDecoder`` of random weights: swiglu MLP, the layers' default configuration."""
    g = torch.Generator().manual_seed(d)
    rn = lambda *s, scale=1.0: torch.randn(*s, generator=g) * scale
    cfg = dict(d_state=S, discretization="ou", zero_process_noise=False, clip_value=None, obs_var_min=1e-4, obs_var_max=None,
               value_rank="full", qk_norm=True, use_conv=True, conv_kernel_size=4, conv_activation="silu", use_gating=True,
               gating_activation="silu", use_lambda_skip=True, return_variance=False, decode_from_prior=False)
    w = {"embedding.weight": rn(vocab, d).to(dtype), "lm_head.weight": rn(vocab, d, scale=d ** -0.5).to(dtype),
         "norm_f.weight": torch.ones(d, dtype=dtype)}
    for i in range(layers):
        b, m = f"blocks.{i}.", f"blocks.{i}.mixer."
        w.update({m + "in_proj.weight": rn(2 * M, d, scale=d ** -0.5).to(dtype),
                  m + "sensor_proj.weight": rn(2 * M + 2 * S, M, scale=M ** -0.5).to(dtype),
                  m + "out_proj.weight": rn(d, M, scale=M ** -0.5).to(dtype), m + "conv.weight": rn(M, 1, 4, scale=0.5),
                  m + "conv.bias": rn(M, scale=0.1), m + "delta": rn(M, S) - 4, m + "lambda_log": rn(M, S, scale=0.1),
                  m + "process_noise": torch.full((M, S), 0.01), m + "lambda_skip": torch.tensor(-1.0),
                  b + "mixer_norm.weight": torch.ones(d, dtype=dtype), b + "mlp_norm.weight": torch.ones(d, dtype=dtype),
                  b + "mlp.w12.weight": rn(4 * d, d, scale=d ** -0.5).to(dtype), b + "mlp.w3.weight": rn(d, 2 * d, scale=(2 * d) ** -0.5).to(dtype)})
    return kla_b200.ModelDecoder(w, [cfg] * layers, dict(n_layers=layers, norm_eps=1e-6, mlp="swiglu", logit_softcap=None))


def test_a_model_on_the_cpu_is_refused_not_served():
    dec = tiny_model()
    ids = torch.zeros(2, 3, dtype=torch.long)
    for call in (lambda: dec.prefill(ids), lambda: dec.step(ids[:, 0], dec.init_state(2, "cpu")), lambda: dec.generate(ids, 4),
                 lambda: dec.generate(ids, 1), lambda: dec.generate(ids, 4, use_graph=False)):
        with pytest.raises(NotImplementedError, match="CUDA"):
            call()


def test_a_kept_decode_step_covers_everything_it_reads(monkeypatch):
    """The captured step is taken again only for the tensors, layouts, settings and modes it was captured with."""
    made = []

    class Graph:
        def __init__(self, *args):
            made.append(args)
            self.done = self

        release = synchronize = lambda self: None

    monkeypatch.setattr(decode, "_TokenGraph", Graph)
    dec = tiny_model(layers=2)

    def captures(call=lambda: None):
        n = len(made)
        call()
        for _ in range(2):
            with dec._token_graph(2, torch.device("cpu"), torch.float32, True):
                pass
        return len(made) - n

    assert captures() == 1 and captures() == 0
    kept = []  # a freed tensor's address could come back with its successor

    def replace(get, put, name):
        kept.append(get(name))
        put(name, kept[-1].clone())

    for layer in dec.layers:
        for name in ("a_bar", "p_bar", "skip", "conv_w", "conv_b"):
            assert captures(lambda: replace(layer.__getattribute__, layer.__setattr__, name)) == 1, name
        for name in ("in_proj.weight", "sensor_proj.weight", "out_proj.weight"):
            assert captures(lambda: replace(layer.w.__getitem__, layer.w.__setitem__, name)) == 1, name
    for name in [n for n in dec.w if ".mixer." not in n]:
        assert captures(lambda: replace(dec.w.__getitem__, dec.w.__setitem__, name)) == 1, name
    w = dec.w["lm_head.weight"]
    assert captures(lambda: dec.w.update({"lm_head.weight": w[:-1]})) == 1  # the same address, another shape
    assert captures(lambda: dec.cfg.update(norm_eps=1e-5)) == 1
    assert captures(lambda: dec.layers[1].cfg.update(obs_var_min=1e-3)) == 1
    with torch.inference_mode():  # tensors made in this mode cannot be written outside it
        assert captures() == 1
    assert captures() == 1


@needs_ref
def test_from_layer_reads_a_reference_layer():
    sys.path.insert(0, REF_SRC)
    try:
        import kla

        torch.manual_seed(0)
        layer = kla.KLALayer(32, kla.KLAConfig(d_state=8, lambda_skip_mode="vector"))
        dec = kla_b200.LayerDecoder.from_layer(layer)
        a_bar, p_bar = layer._compute_aq()
        torch.testing.assert_close(dec.a_bar, a_bar.detach())
        torch.testing.assert_close(dec.p_bar, p_bar.detach())
        assert dec.skip.shape == (layer.d_inner,) and dec.conv_w.shape == (layer.d_inner, 4)
    finally:
        sys.path.remove(REF_SRC)


# ----------------------------------------------------------------------- GPU

def _run(name, dtype, steps=3):
    dev = torch.device("cuda:0")
    z, weights, config = load(name)
    weights = {k: (v.to(dtype) if k.split(".")[0] in ("in_proj", "sensor_proj", "out_proj", "value_expand", "var_expand")
                   else v) for k, v in weights.items()}
    dec = kla_b200.LayerDecoder(weights, config).to(dev)
    conv = torch.from_numpy(z["conv0"]).to(dev, dtype) if "conv0" in z else None
    state = (conv, torch.from_numpy(z["lam0"]).to(dev), torch.from_numpy(z["eta0"]).to(dev))
    outs = []
    for t in range(steps):
        res = dec.step(torch.from_numpy(z["x"][t]).to(dev, dtype), state)
        outs.append(tuple(r.float().cpu() for r in (res if isinstance(res, tuple) else (res,))))
        outs[-1] += tuple(None if s is None else s.float().cpu().clone() for s in state)
    return z, config, outs


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_decode_matches_reference_layer_f32(name):
    z, config, outs = _run(name, torch.float32)
    for t, got in enumerate(outs):
        n_out = 2 if config["return_variance"] else 1
        torch.testing.assert_close(got[0], torch.from_numpy(z[f"out{t}"]), rtol=1e-4, atol=1e-5, msg=lambda m: f"out{t}: {m}")
        if n_out == 2:
            torch.testing.assert_close(got[1], torch.from_numpy(z[f"outvar{t}"]), rtol=1e-4, atol=1e-5)
        conv, lam, eta = got[n_out:]
        if conv is not None:
            torch.testing.assert_close(conv, torch.from_numpy(z[f"conv{t + 1}"]), rtol=1e-5, atol=1e-6)
        torch.testing.assert_close(lam, torch.from_numpy(z[f"lam{t + 1}"]), rtol=2e-5, atol=1e-6)
        torch.testing.assert_close(eta, torch.from_numpy(z[f"eta{t + 1}"]), rtol=2e-5, atol=2e-6)
    L = import_module("kalman-linear-attention_b200._lib")
    assert L.device_status() == 0


@pytest.mark.gpu
def test_decode_bf16_activations_stay_close():
    z, config, outs = _run("default", torch.bfloat16)
    for t, got in enumerate(outs):
        ref = torch.from_numpy(z[f"out{t}"])
        assert (got[0] - ref).abs().max() <= 3e-2 * (1.0 + ref.abs().max())


@pytest.mark.gpu
def test_decode_step_is_graph_capturable():
    dev = torch.device("cuda:0")
    z, weights, config = load("default")
    dec = kla_b200.LayerDecoder(weights, config).to(dev)

    def fresh():
        return (torch.from_numpy(z["conv0"]).to(dev), torch.from_numpy(z["lam0"]).to(dev), torch.from_numpy(z["eta0"]).to(dev))

    x = torch.from_numpy(z["x"][0]).to(dev)
    state = fresh()
    dec.step(x, state)  # warm-up outside capture (library handles, lazy loads)
    state = fresh()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = dec.step(x, state)
    torch.cuda.current_stream().wait_stream(s)
    for buf, src in zip(state, fresh()):
        buf.copy_(src)
    g.replay()
    torch.cuda.synchronize()
    torch.testing.assert_close(out.cpu(), torch.from_numpy(z["out0"]), rtol=1e-4, atol=1e-5)
    torch.testing.assert_close(state[1].cpu(), torch.from_numpy(z["lam1"]), rtol=2e-5, atol=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("name", CASES)
def test_prefill_then_decode_matches_reference_layer(name):
    """The whole inference route: prefill through the scan kernels (sensor prologue and skip/gate
    epilogue inside), then token-by-token decode from the state the prefill left."""
    dev = torch.device("cuda:0")
    z, weights, config = load(name)
    dec = kla_b200.LayerDecoder(weights, config).to(dev)
    pre, state = dec.prefill(torch.from_numpy(z["x0"]).to(dev))
    outs = pre if isinstance(pre, tuple) else (pre,)
    torch.testing.assert_close(outs[0].cpu(), torch.from_numpy(z["pre_out"]), rtol=1e-4, atol=2e-5)
    if config["return_variance"]:
        torch.testing.assert_close(outs[1].cpu(), torch.from_numpy(z["pre_outvar"]), rtol=1e-4, atol=2e-5)
    if "conv0" in z:
        torch.testing.assert_close(state[0].cpu(), torch.from_numpy(z["conv0"]), rtol=1e-5, atol=1e-6)
    torch.testing.assert_close(state[1].cpu(), torch.from_numpy(z["lam0"]), rtol=5e-5, atol=1e-5)
    torch.testing.assert_close(state[2].cpu(), torch.from_numpy(z["eta0"]), rtol=5e-5, atol=1e-5)
    for t in range(3):
        res = dec.step(torch.from_numpy(z["x"][t]).to(dev), state)
        out = res[0] if isinstance(res, tuple) else res
        torch.testing.assert_close(out.cpu(), torch.from_numpy(z[f"out{t}"]), rtol=2e-4, atol=3e-5)
    torch.testing.assert_close(state[1].cpu(), torch.from_numpy(z["lam3"]), rtol=1e-4, atol=1e-5)


# ------------------------------------------------------------ causal convolution over a sequence, forward + backward

def _conv_module_math(x, weight, bias, state, act):
    """CausalConv1d.forward (src/kla/layers/common.py:87-96) as plain torch operations."""
    B, L, D = x.shape
    K = weight.shape[-1]
    x_t = x.transpose(1, 2)
    if state is None:
        state = torch.zeros(B, D, K - 1, device=x.device, dtype=x.dtype)
    x_pad = torch.cat((state.to(x_t.dtype), x_t), dim=-1)
    y = torch.nn.functional.conv1d(x_pad, weight, bias, groups=D)
    return getattr(torch.nn.functional, act)(y).transpose(1, 2), x_pad[..., x_pad.shape[-1] - (K - 1):]


@pytest.mark.gpu
@pytest.mark.parametrize("B,L,D,K,act,with_state,with_bias", [
    (2, 200, 96, 4, "silu", False, True),     # the layer's defaults; L not a multiple of the kernels' chunks
    (1, 64, 130, 4, "gelu", True, True),      # carried window, channels not a multiple of the block
    (3, 129, 32, 8, "relu", True, False),     # most taps, no bias
    (2, 2, 16, 4, "silu", True, True),        # sequence shorter than the window
    (2, 33, 20, 1, "silu", False, True),      # one tap: no window at all
    (2, 70, 64, 2, "gelu", False, False),
])
def test_causal_conv_forward_backward(B, L, D, K, act, with_state, with_bias):
    layer = import_module("kalman-linear-attention_b200.layer")
    g = torch.Generator().manual_seed(B * 1000 + L + K)
    # x as the layer hands it over: one half of a wider projection, i.e. a view with a row stride of 2 D
    wide = torch.randn(B, L, 2 * D, generator=g).cuda()
    weight = (torch.randn(D, 1, K, generator=g) * 0.5).cuda().requires_grad_(True)
    bias = torch.randn(D, generator=g).cuda().requires_grad_(True) if with_bias else None
    state = torch.randn(B, D, K - 1, generator=g).cuda() if with_state else None
    dz = torch.randn(B, L, D, generator=g).cuda()

    def run(fn):
        w2 = wide.clone().requires_grad_(True)
        z, st = fn(w2[..., :D], weight, bias, state, act)
        grads = torch.autograd.grad(z, [w2, weight] + ([bias] if with_bias else []), dz)
        return [z.detach(), st.detach()] + [t.detach() for t in grads]

    got = run(layer.causal_conv_b200)
    want = run(_conv_module_math)
    names = ["z", "new_state", "dx", "dweight", "dbias"]
    for n, a_, b_ in zip(names, got, want):
        assert a_.shape == b_.shape, n
        torch.testing.assert_close(a_, b_, rtol=2e-5, atol=2e-5, msg=lambda m, n=n: f"{n}: {m}")


@pytest.mark.gpu
def test_causal_conv_bf16_tracks_float32():
    layer = import_module("kalman-linear-attention_b200.layer")
    g = torch.Generator().manual_seed(5)
    B, L, D, K = 2, 300, 256, 4
    x32 = torch.randn(B, L, D, generator=g).cuda()
    weight = (torch.randn(D, 1, K, generator=g) * 0.5).cuda().requires_grad_(True)
    bias = torch.randn(D, generator=g).cuda().requires_grad_(True)
    dz = torch.randn(B, L, D, generator=g).cuda()
    outs = {}
    for dt in (torch.float32, torch.bfloat16):
        x = x32.to(dt).requires_grad_(True)
        z, _ = layer.causal_conv_b200(x, weight, bias, None, "silu")
        assert z.dtype == dt
        outs[dt] = [z.float().detach()] + [t.float() for t in torch.autograd.grad(z, [x, weight, bias], dz.to(dt))]
    for a_, b_ in zip(outs[torch.bfloat16], outs[torch.float32]):
        assert ((a_ - b_).abs().max() / (b_.abs().max() + 1e-6)).item() < 2e-2


# ------------------------------------------------------------ what the kernels are not given

@pytest.mark.gpu
def test_types_without_a_kernel_are_refused():
    layer = import_module("kalman-linear-attention_b200.layer")
    for dtype in (torch.float16, torch.float64):
        dec = tiny_model(dtype=dtype).to("cuda")
        ids = torch.zeros(2, 3, dtype=torch.long, device="cuda")
        for call in (lambda: dec.step(ids[:, 0], dec.init_state(2, "cuda", dtype)), lambda: dec.prefill(ids), lambda: dec.generate(ids, 3),
                     lambda: dec.layers[0].step(torch.zeros(2, 32, device="cuda", dtype=dtype), dec.layers[0].init_state(2, "cuda", dtype)),
                     lambda: layer.causal_conv_b200(torch.zeros(1, 8, 32, device="cuda", dtype=dtype), torch.zeros(32, 1, 4, device="cuda"), None)):
            with pytest.raises(NotImplementedError, match="float32 or bfloat16"):
                call()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_a_state_that_does_not_fit_the_token_is_refused(dtype):
    dec = tiny_model(dtype=dtype).to("cuda").layers[0]
    M, S, B = dec.M, dec.S, 3
    x = torch.zeros(B, 32, device="cuda", dtype=dtype)
    good = dec.init_state(B, "cuda", dtype)
    dec.step(x, good)
    conv, lam, eta = good
    other = torch.bfloat16 if dtype == torch.float32 else torch.float32
    wide = torch.ones(B, 2, M, S, device="cuda")
    for bad in (dec.init_state(B - 1, "cuda", dtype), (conv.to(other), lam, eta), (conv[..., :2], lam, eta), (None, lam, eta),
                (conv, lam.double(), eta), (conv, wide[:, 0], eta), (conv, lam, eta[:, :-1].contiguous()), (conv, lam.cpu(), eta)):
        with pytest.raises(ValueError):
            dec.step(x, bad)
    dec.w = dict(dec.w, **{"in_proj.weight": dec.w["in_proj.weight"][:M]})
    with pytest.raises(ValueError, match="in_proj"):
        dec.step(x, good)


@pytest.mark.gpu
def test_decode_under_autocast_follows_float32():
    """Autocast gives float32 activations bfloat16 projections. Each of a layer's three rounds its operands and its result
    (2^-9 of their size); what is between them does not enlarge that, so 3e-2 of the output's size covers it."""
    dec = tiny_model(d=64, M=128).to("cuda").layers[0]
    g = torch.Generator().manual_seed(3)
    prompt, x = torch.randn(2, 20, 64, generator=g).cuda(), torch.randn(2, 64, generator=g).cuda()
    want, state = dec.prefill(prompt)
    want_step = dec.step(x, state)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        got, state_a = dec.prefill(prompt)
        got_step = dec.step(x, state_a)
    assert [t.dtype for t in state_a] == [t.dtype for t in state]
    for a, b in ((got, want), (got_step, want_step)):
        assert (a.float() - b).abs().max() <= 3e-2 * b.abs().max()
    torch.testing.assert_close(state_a[0], state[0], rtol=2e-2, atol=2e-2 * state[0].abs().mean().item())


@pytest.mark.gpu
@pytest.mark.parametrize("use_conv", [True, False])
def test_a_layer_uses_the_weights_the_kernel_in_front_of_it_writes(use_conv):
    """The decode projections let their successor start before they have stored anything. Here one of them produces the
    weights of the layer whose token comes next."""
    lib = import_module("kalman-linear-attention_b200._lib")
    dec = tiny_model(dtype=torch.bfloat16).to("cuda").layers[0]
    if not use_conv:
        dec.cfg["use_conv"], dec.conv_w, dec.conv_b = False, None, None
    g = torch.Generator(device="cuda").manual_seed(1)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, source = rn(4, 32), rn(128, 8192) * 8192 ** -0.5
    in_shape = dec.w["in_proj.weight"].shape
    for _ in range(20):
        seed = rn(32, 8192)
        torch.cuda.synchronize()
        made = lib.host().project(seed, source, None, None, 0.0, None)  # [32, 128]
        dec.w = dict(dec.w, **{"in_proj.weight": made.view(in_shape)})
        got = dec.step(x, dec.init_state(4, "cuda", torch.bfloat16))
        torch.cuda.synchronize()
        assert torch.equal(got, dec.step(x, dec.init_state(4, "cuda", torch.bfloat16)))


@pytest.mark.gpu
def test_generated_ids_are_int64_for_any_count():
    dec = tiny_model().to("cuda")
    ids = torch.tensor([[1, 2, 3], [4, 5, 6]], device="cuda")
    want = dec.generate(ids, 5)
    for dtype in (torch.int32, torch.int64):
        for new in (1, 5):
            got = dec.generate(ids.to(dtype), new)
            assert got.dtype == torch.int64 and torch.equal(got, want[:, :3 + new])


@pytest.mark.gpu
def test_a_kept_step_on_another_stream_keeps_its_buffers_until_it_is_done():
    """The kept step's buffers belong to the stream of the call that captured it. A later call replays it on another
    stream; the decoder is dropped while that stream still has it all to do, and the first stream asks for memory."""
    dec = tiny_model(d=64, M=256, layers=2).to("cuda")
    ids = torch.arange(12, device="cuda").view(2, 6)
    want = dec.generate(ids, 24)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(40_000_000)  # 20 ms
        got = dec.generate(ids, 24)
    shapes = {t.shape for layer in dec._slot.graph.state for t in layer} | {dec._slot.graph.token.shape}
    weights = [dec.w, *(dict(layer.__dict__) for layer in dec.layers)]  # the caller's to keep
    del dec
    taken = [torch.full(s, 1e9, device="cuda") for s in shapes for _ in range(8)]
    torch.cuda.synchronize()
    assert torch.equal(got, want) and taken and weights
