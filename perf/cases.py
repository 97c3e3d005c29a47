"""The calls a user of this package makes, as timeable cases.

``listed()`` names one case for each way the package is used: single-token decode, prompt prefill, generation with a
whole model, inference over one sequence, and training of the scan at small, ragged, ordinary and long shapes. ``draw``
gives further cases from the same ranges. A case is prepared once (``prepare``: inputs on the GPU, weights, decoders)
and then run any number of times (``run``: one pass through the public entry points).
"""

import math

import torch
import torch.nn.functional as F

import kla_b200

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
TAPS = 4  # taps of the layer's causal convolution

LAYER_CONFIG = dict(
    discretization="ou", zero_process_noise=False, clip_value=None, obs_var_min=1e-4, obs_var_max=None,
    value_rank="full", qk_norm=True, use_conv=True, conv_kernel_size=TAPS, conv_activation="silu", use_gating=True,
    gating_activation="silu", use_lambda_skip=True, return_variance=False, decode_from_prior=False)


def listed():
    return [
        # one decode step of one small layer's filter, as the reference layer calls it per token: latency only
        dict(name="step_small", kind="step", B=4, M=1024, S=16, dtype="f32"),
        # one token of one layer at serving batch (d_model 1024, 2048 channels, bf16 activations, f32 state)
        dict(name="layer_step", kind="layer_step", B=32, d_model=1024, S=16, dtype="bf16"),
        # a whole 12-layer model answering a batch of prompts, greedy
        dict(name="generate", kind="generate", B=8, prompt=512, new=64, d_model=768, layers=12, vocab=50304, S=16,
             dtype="bf16"),
        # a long prompt through one layer in inference, state kept for decode
        dict(name="prefill", kind="prefill", B=4, L=8192, d_model=1024, S=16, dtype="bf16"),
        # inference over ONE sequence whose length is whatever the text's length is
        dict(name="scan_one_sequence", kind="scan", B=1, L=1501, M=1536, S=16, dtype="f32"),
        # training: the example layer's scan (d_model 512, batch 2, T 1024)
        dict(name="train_small", kind="train", B=2, L=1024, M=1024, S=16, dtype="f32", carry=False),
        # training on a batch whose sizes divide into nothing
        dict(name="train_ragged", kind="train", B=3, L=1537, M=1001, S=16, dtype="f32", carry=True),
        # training at the headline shape
        dict(name="train_headline", kind="train", B=8, L=4096, M=1024, S=16, dtype="f32", carry=False),
        # training on long contexts in bf16, continued from a carried state
        dict(name="train_long", kind="train", B=2, L=65536, M=4096, S=16, dtype="bf16", carry=True),
        # training with a larger filter state per channel
        dict(name="train_wide_state", kind="train", B=4, L=2048, M=512, S=64, dtype="f32", carry=False),
        # a training step of the 768-wide layer between its projections: convolution, sensor prologue, scan, skip, gate
        dict(name="train_layer", kind="train_layer", B=16, L=2048, M=1536, S=16, dtype="bf16"),
        # the raw scan pair over materialised coefficients, both directions
        dict(name="raw_pair", kind="raw_pair", B=2, L=4096, M=1024, S=16, dtype="f32"),
    ]


def _log(rng, lo, hi):
    """A size between ``lo`` and ``hi``, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _width(rng, lo, hi):
    """A channel count: mostly a multiple of 64 as layers have it, sometimes any number."""
    n = _log(rng, lo, hi)
    return n if rng.random() < 0.3 else max(64, n // 64 * 64)


def draw(rng):
    kind = rng.choice(["step", "layer_step", "generate", "prefill", "scan", "train", "train", "train_long",
                       "train_layer", "raw_pair"])
    S = rng.choice([16, 16, 16, 8, 32, 64])
    dtype = rng.choice(["f32", "bf16"])
    if kind == "step":
        return dict(kind=kind, B=_log(rng, 1, 256), M=_width(rng, 256, 4096), S=S, dtype=dtype)
    if kind == "layer_step":
        return dict(kind=kind, B=_log(rng, 1, 64), d_model=_log(rng, 256, 1024) // 8 * 8, S=rng.choice([8, 16, 32]),
                    dtype=dtype)
    if kind == "generate":
        return dict(kind=kind, B=_log(rng, 1, 8), prompt=_log(rng, 16, 512), new=_log(rng, 8, 64),
                    d_model=_log(rng, 128, 768) // 16 * 16, layers=rng.randint(2, 12),
                    vocab=rng.choice([512, 8192, 32000, 50304]), S=16, dtype="bf16")
    if kind == "prefill":
        d = _log(rng, 256, 1024) // 8 * 8
        B = _log(rng, 1, 8)
        return dict(kind=kind, B=B, L=_log(rng, 64, min(8192, 4 * 8192 * 1024 // (B * d))), d_model=d, S=16,
                    dtype="bf16")
    if kind == "scan":
        B = _log(rng, 1, 4)
        M = _width(rng, 256, 4096)
        return dict(kind=kind, B=B, L=_log(rng, 32, min(8192, 2 ** 25 // (B * M))), M=M, S=16, dtype=dtype)
    if kind == "train":
        B = _log(rng, 1, 16)
        M = _width(rng, 128, 2048)
        top = 2 ** 25 * 16 // (B * M * S)
        return dict(kind=kind, B=B, L=_log(rng, 64, max(65, min(8192, top))), M=M, S=S, dtype=dtype,
                    carry=rng.random() < 0.5)
    if kind == "train_long":
        M = _log(rng, 512, 4096) // 64 * 64
        return dict(kind="train", B=rng.choice([1, 2]), L=_log(rng, 12288, 65536), M=M, S=16, dtype="bf16",
                    carry=rng.random() < 0.5)
    if kind == "train_layer":
        B = _log(rng, 1, 16)
        M = _log(rng, 256, 2048) // 16 * 16
        return dict(kind=kind, B=B, L=_log(rng, 128, min(4096, 16 * 2048 * 1536 // (B * M))), M=M, S=16, dtype=dtype)
    B = _log(rng, 1, 8)
    M = _width(rng, 64, 1024)
    return dict(kind="raw_pair", B=B, L=_log(rng, 64, min(4096, 2 * 4096 * 1024 // (B * M))), M=M, S=16, dtype="f32")


def _random(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *shape, scale=1.0: torch.randn(*shape, generator=g, device="cuda").mul_(scale)


def _layer_weights(rn, d_model, S, dtype):
    M = 2 * d_model
    return {
        "in_proj.weight": rn(2 * M, d_model, scale=d_model ** -0.5).to(dtype),
        "sensor_proj.weight": rn(2 * M + 2 * S, M, scale=M ** -0.5).to(dtype),
        "out_proj.weight": rn(d_model, M, scale=M ** -0.5).to(dtype),
        "conv.weight": rn(M, 1, TAPS, scale=0.5), "conv.bias": rn(M, scale=0.02),
        "delta": rn(M, S) - 4.0, "lambda_log": rn(M, S, scale=0.1),
        "process_noise": torch.full((M, S), 0.01, device="cuda"),
        "lambda_skip": torch.tensor(-1.0, device="cuda"),
    }


def _prepare_decode(case, rn, dtype):
    B, d, S = case["B"], case["d_model"], case["S"]
    config = dict(LAYER_CONFIG, d_state=S)
    if case["kind"] != "generate":
        dec = kla_b200.LayerDecoder(_layer_weights(rn, d, S, dtype), config).to("cuda")
        if case["kind"] == "prefill":
            return dict(dec=dec, x=rn(B, case["L"], d).to(dtype))
        conv, lam, eta = dec.init_state(B, "cuda", dtype)
        conv.copy_(rn(*conv.shape))
        lam.copy_(F.softplus(rn(*lam.shape)) + 0.5)
        eta.copy_(rn(*eta.shape))
        return dict(dec=dec, x=rn(B, d).to(dtype), state=(conv, lam, eta))
    V, n, hidden = case["vocab"], case["layers"], 8 * d // 3 // 16 * 16
    emb = rn(V, d)
    # a trained model is sure of most of its next tokens: the head's row of the token that follows t looks for t
    follows = torch.argsort(rn(V))
    head = torch.empty_like(emb)
    head[follows] = emb
    weights = {"embedding.weight": emb.to(dtype), "lm_head.weight": head.mul_(d ** -0.5).to(dtype),
               "norm_f.weight": torch.ones(d, device="cuda", dtype=dtype)}
    for i in range(n):
        pre = f"blocks.{i}."
        weights.update({pre + "mixer." + k: v for k, v in _layer_weights(rn, d, S, dtype).items()})
        weights[pre + "mixer_norm.weight"] = torch.ones(d, device="cuda", dtype=dtype)
        weights[pre + "mlp_norm.weight"] = torch.ones(d, device="cuda", dtype=dtype)
        weights[pre + "mlp.w12.weight"] = rn(2 * hidden, d, scale=d ** -0.5).to(dtype)
        weights[pre + "mlp.w3.weight"] = rn(d, hidden, scale=hidden ** -0.5).to(dtype)
    model = dict(n_layers=n, norm_eps=1e-6, mlp="swiglu", logit_softcap=None)
    ids = torch.argsort(rn(B, V), dim=1)[:, :1].expand(B, case["prompt"]).contiguous()
    ids = (ids + torch.arange(case["prompt"], device="cuda") * 7919) % V
    return dict(dec=kla_b200.ModelDecoder(weights, [config] * n, model), ids=ids, new=case["new"])


def _prepare_raw(case, rn):
    B, L, M, S = (case[n] for n in ("B", "L", "M", "S"))
    a2 = torch.sigmoid(rn(M, S)).square()
    p = F.softplus(rn(M, S))
    phi = rn(B, L, M, S).square_().mul_(1.0 / S)
    ins = [1.0 + p * phi, a2 * phi, p.expand(B, L, M, S).contiguous(), a2.expand(B, L, M, S).contiguous(),
           torch.sigmoid(rn(B, L, M, S)), rn(B, L, M, S)]
    return dict(ins=[t.requires_grad_() for t in ins], grads=[rn(B, L, M, S), rn(B, L, M, S)])


def prepare(case, seed):
    rn, kind, dtype = _random(seed), case["kind"], DTYPES[case["dtype"]]
    if kind in ("layer_step", "prefill", "generate"):
        return dict(_prepare_decode(case, rn, dtype), kind=kind)
    if kind == "raw_pair":
        return dict(_prepare_raw(case, rn), kind=kind)
    B, M, S = case["B"], case["M"], case["S"]
    rows = (B,) if kind == "step" else (B, case["L"])
    a = torch.sigmoid(rn(M, S))
    p = F.softplus(rn(M, S))
    if kind == "train_layer":
        leaves = dict(projected=rn(*rows, 2 * M).to(dtype), sensors=rn(*rows, 2 * M + 2 * S).to(dtype),
                      weight=rn(M, 1, TAPS, scale=0.5), bias=rn(M, scale=0.02), a=a, p=p,
                      skip=torch.tensor(-1.0, device="cuda") + rn(1, scale=0.1)[0])
        return dict(kind=kind, M=M, S=S, dtype=dtype, leaves={n: t.requires_grad_() for n, t in leaves.items()},
                    grads=[rn(*rows, M).to(dtype), rn(*rows, M).to(dtype)])
    v = rn(*rows, M).to(dtype)
    lambda_v = F.softplus(rn(*rows, M)).reciprocal_().to(dtype)
    k = F.normalize(rn(*rows, S), dim=-1).to(dtype)
    q = F.normalize(rn(*rows, S), dim=-1).to(dtype)
    ins = [v, lambda_v, k, q, a, p]
    carried = None
    if kind == "step" or case.get("carry"):
        carried = (F.softplus(rn(B, M, S)) + 0.5, rn(B, M, S))
    grads = None
    if kind == "train":
        ins = [t.requires_grad_() for t in ins]
        grads = [rn(*rows, M).to(dtype), rn(*rows, M).to(dtype)]
        if carried is not None:
            carried = tuple(t.requires_grad_() for t in carried)
            grads += [rn(B, M, S, scale=0.1), rn(B, M, S, scale=0.1)]
    return dict(kind=kind, ins=ins, carried=carried, grads=grads, dtype=dtype)


def _run_train_layer(s):
    w, M, S = s["leaves"], s["M"], s["S"]
    z, gate = w["projected"].chunk(2, dim=-1)
    z, window = kla_b200.layer.causal_conv_b200(z, w["weight"], w["bias"], None, "silu")
    v, log_var, k, q = torch.split(w["sensors"], [M, M, S, S], dim=-1)
    k, q = F.normalize(k, dim=-1), F.normalize(q, dim=-1)
    y, y_var, st = kla_b200.kla_scan_b200(
        v, log_var, k, q, w["a"], w["p"], out_dtype=s["dtype"], log_variance=(1e-4, None),
        epilogue=dict(z=z, lambda_skip=w["skip"], gate=gate, gate_activation="silu"))
    return [y, y_var, st.lam, st.eta, window, *torch.autograd.grad([y, y_var], list(w.values()), s["grads"])]


def run(s):
    kind = s["kind"]
    if kind == "step":
        with torch.no_grad():
            y, y_var, st = kla_b200.kla_step_b200(*s["ins"], s["carried"])
        return [y, y_var, st.lam, st.eta]
    if kind == "layer_step":
        with torch.no_grad():
            return [s["dec"].step(s["x"], s["state"]), *s["state"]]
    if kind == "prefill":
        out, state = s["dec"].prefill(s["x"])
        return [out, *state]
    if kind == "generate":
        return [s["dec"].generate(s["ids"], s["new"])]
    if kind == "scan":
        with torch.no_grad():
            y, y_var, st = kla_b200.kla_scan_b200(*s["ins"], out_dtype=s["dtype"])
        return [y, y_var, st.lam, st.eta]
    if kind == "train_layer":
        return _run_train_layer(s)
    if kind == "raw_pair":
        lam = kla_b200.mobius_scan_b200(*s["ins"][:4])
        eta = kla_b200.affine_scan_b200(*s["ins"][4:])
        return [lam, eta, *torch.autograd.grad([lam, eta], s["ins"], s["grads"])]
    y, y_var, st = kla_b200.kla_scan_b200(*s["ins"], initial_state=s["carried"], out_dtype=s["dtype"])
    outs, leaves = [y, y_var], list(s["ins"])
    if s["carried"] is not None:
        outs += [st.lam, st.eta]
        leaves += s["carried"]
    return [y, y_var, st.lam, st.eta, *torch.autograd.grad(outs, leaves, s["grads"])]


def work(case):
    """Inputs read once and outputs written once; a filter step of one (channel, state) pair is 16 operations and its
    adjoint 50; a projection is 2 per weight and row."""
    kind, B, S = case["kind"], case["B"], case["S"]
    e = 4 if case["dtype"] == "f32" else 2
    if kind in ("layer_step", "prefill", "generate"):
        d = case["d_model"]
        M = 2 * d
        weights = 2 * M * d + M * (2 * M + 2 * S) + M * d
        if kind == "generate":
            n, hidden = case["layers"], 8 * d // 3 // 16 * 16
            weights = n * (weights + 3 * hidden * d)
            head = case["vocab"] * d
            rows = B * (case["prompt"] + case["new"] - 1)
            # the prompt's pass reads every weight once, and so does each token after it
            return {"bytes": case["new"] * (e * (weights + head) + 16 * n * B * M * S) + 8 * rows,
                    "flops": 2 * rows * weights + 2 * B * case["new"] * head + 16 * n * rows * M * S}
        rows = B * (1 if kind == "layer_step" else case["L"])
        return {"bytes": e * (weights + 2 * rows * d) + 8 * M * S + 16 * B * M * S,
                "flops": 2 * rows * weights + 16 * rows * M * S}
    M = case["M"]
    rows = B * (1 if kind == "step" else case["L"])
    if kind == "raw_pair":
        return {"bytes": 4 * rows * M * S * 16, "flops": 24 * rows * M * S}
    if kind in ("step", "scan"):
        state = 4 * B * M * S * (4 if kind == "step" else 2)
        outs = 4 if kind == "step" else e
        return {"bytes": rows * (2 * M + 2 * S) * e + rows * 2 * M * outs + 8 * M * S + state,
                "flops": 16 * rows * M * S}
    if kind == "train_layer":
        return {"bytes": rows * e * (2 * (4 * M + 2 * S) + 4 * M) + 16 * M * S + 8 * B * M * S,
                "flops": 66 * rows * M * S + 60 * rows * M}
    return {"bytes": rows * e * (8 * M + 4 * S) + 16 * M * S + 4 * B * M * S * (8 if case["carry"] else 2),
            "flops": 66 * rows * M * S}


def tolerance(case):
    if case["kind"] == "generate":
        return {"rel": 0.0, "differ": 0.005}  # whole tokens
    # f32: sums over thousands of steps and channels, in another order; bf16: its rounding of inputs and results
    return {"rel": 1e-4} if case["dtype"] == "f32" else {"rel": 1e-2}
