"""Prompt and token loop of a whole model (``ModelDecoder``) in bfloat16 against a restatement of the model in plain torch
operations, without the reference package; and the captured decode step that ``generate`` keeps between calls."""

import os
import sys
import threading

import pytest
import torch
import torch.nn.functional as F

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
import kla_b200  # noqa: E402

pytestmark = pytest.mark.gpu
EPS = 1e-6
CONFIG = dict(discretization="ou", zero_process_noise=False, clip_value=None, obs_var_min=1e-4, obs_var_max=None,
              value_rank="full", qk_norm=True, use_conv=True, conv_kernel_size=4, conv_activation="silu", use_gating=True,
              gating_activation="silu", use_lambda_skip=True, return_variance=False, decode_from_prior=False)


def model_weights(d, layers, vocab, S=16, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s, scale=1.0: torch.randn(*s, generator=g, device="cuda") * scale
    bf = lambda *s: rn(*s, scale=s[-1] ** -0.5).bfloat16()
    M = 2 * d
    w = {"embedding.weight": rn(vocab, d).bfloat16(), "lm_head.weight": bf(vocab, d), "norm_f.weight": (1 + rn(d, scale=0.1)).bfloat16()}
    for i in range(layers):
        b, m = f"blocks.{i}.", f"blocks.{i}.mixer."
        w.update({m + "in_proj.weight": bf(2 * M, d), m + "sensor_proj.weight": bf(2 * M + 2 * S, M), m + "out_proj.weight": bf(d, M),
                  m + "conv.weight": rn(M, 1, 4, scale=0.5), m + "conv.bias": rn(M, scale=0.1), m + "delta": rn(M, S) - 4,
                  m + "lambda_log": rn(M, S, scale=0.1), m + "process_noise": torch.full((M, S), 0.01, device="cuda"),
                  m + "lambda_skip": torch.tensor(-1.0, device="cuda"), b + "mixer_norm.weight": (1 + rn(d, scale=0.1)).bfloat16(),
                  b + "mlp_norm.weight": (1 + rn(d, scale=0.1)).bfloat16(), b + "mlp.w12.weight": bf(4 * d, d), b + "mlp.w3.weight": bf(d, 2 * d)})
    return w


def decoder(w, layers, S=16):
    return kla_b200.ModelDecoder(w, [dict(CONFIG, d_state=S)] * layers, dict(n_layers=layers, norm_eps=EPS, mlp="swiglu", logit_softcap=None))


@torch.no_grad()
def restated(w, layers, ids, act, filt):
    """Logits [B, L, vocab] of the model, one token at a time: activations, projections and what stands between them as torch
    operations in ``act``, each rounding its result; norms and the filter in ``filt`` (src/kla/models/sequence_model.py:47-98,
    150-173; src/kla/layers/common.py:45-55, 87-122; src/kla/layers/kla_layer.py:199-231, 277-345; src/kla/ops/kla_ops.py:293-331)."""
    B, L = ids.shape
    W = lambda name: w[name].to(act)

    def norm(x, name):
        x = x.to(filt)
        return (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS) * w[name].to(filt)).to(act)

    state = []
    for i in range(layers):
        m = f"blocks.{i}.mixer."
        a = -torch.exp(w[m + "lambda_log"].to(filt))
        delta = F.softplus(w[m + "delta"].to(filt)) + 1e-7
        a_bar, lam_pos = torch.exp(delta * a), a.abs().clamp_min(1e-8)
        p_bar = (w[m + "process_noise"].to(filt).clamp_min(1e-7) / (2 * lam_pos)) * -torch.expm1(-2 * lam_pos * delta)
        M, S = a.shape
        state.append([torch.zeros(B, M, 3, device=ids.device, dtype=act), torch.ones(B, M, S, device=ids.device, dtype=filt),
                      torch.zeros(B, M, S, device=ids.device, dtype=filt), a_bar, p_bar])
    logits = []
    for t in range(L):
        x = F.embedding(ids[:, t], W("embedding.weight"))
        for i, st in enumerate(state):
            b, m = f"blocks.{i}.", f"blocks.{i}.mixer."
            window, lam, eta, a, p = st
            M, S = a.shape
            z, gate = F.linear(norm(x, b + "mixer_norm.weight"), W(m + "in_proj.weight")).chunk(2, dim=-1)
            taps = torch.cat((window, z.unsqueeze(-1)), dim=-1)
            st[0] = taps[..., 1:]
            z = F.silu(((taps.to(filt) * w[m + "conv.weight"].to(filt).squeeze(1)).sum(-1) + w[m + "conv.bias"].to(filt)).to(act))
            v, s, k, q = torch.split(F.linear(z, W(m + "sensor_proj.weight")), [M, M, S, S], dim=-1)
            k, q = (u.to(filt) / u.to(filt).norm(dim=-1, keepdim=True).clamp_min(1e-12) for u in (k, q))
            lv = 1 / (F.softplus(s.to(filt)) + CONFIG["obs_var_min"])
            inv = 1 / (a * a + p * lam)
            st[1] = lam * inv + (lv.unsqueeze(-1) * k.unsqueeze(1) ** 2)
            st[2] = a * inv * eta + (v.to(filt) * lv).unsqueeze(-1) * k.unsqueeze(1)
            y = ((st[2] / st[1]) * q.unsqueeze(1)).sum(-1).to(act)
            y = (y + w[m + "lambda_skip"].to(act) * z) * F.silu(gate)
            x = x + F.linear(y, W(m + "out_proj.weight"))
            g, u = F.linear(norm(x, b + "mlp_norm.weight"), W(b + "mlp.w12.weight")).chunk(2, dim=-1)
            x = x + F.linear(F.silu(g) * u, W(b + "mlp.w3.weight"))
        logits.append(F.linear(norm(x, "norm_f.weight"), W("lm_head.weight")))
    return torch.stack(logits, dim=1)


# narrow and deep, where the largest logits nearly tie; wide; the library's route beyond 16 and beyond 32 rows
@pytest.mark.parametrize("B,d,layers,vocab,prompt,new", [(4, 128, 12, 512, 9, 40), (2, 144, 10, 8192, 17, 24), (8, 768, 2, 8192, 12, 16),
                                                         (20, 768, 2, 512, 6, 12), (40, 256, 4, 512, 6, 12)])
def test_logits_and_tokens_are_as_close_as_torch_operations_come(B, d, layers, vocab, prompt, new):
    """All three see the same tokens, those ``generate`` chose. The error of the bfloat16 kernels' logits against float64 is
    held to that of torch's bfloat16 operations, which round in more places; where the kernels choose another token than
    float64, the two logits lie within that error of each other."""
    w = model_weights(d, layers, vocab)
    dec = decoder(w, layers)
    ids = torch.randint(0, vocab, (B, prompt), generator=torch.Generator().manual_seed(d)).cuda()
    tokens = dec.generate(ids, new)
    assert torch.equal(tokens[:, :prompt], ids) and torch.equal(dec.generate(ids, new, use_graph=False), tokens)
    exact = restated(w, layers, tokens[:, :-1], torch.float64, torch.float64)
    plain = restated(w, layers, tokens[:, :-1], torch.bfloat16, torch.float32).double()
    got, state = dec.prefill(ids)
    got = torch.cat([got, *(dec.step(tokens[:, t], state).unsqueeze(1) for t in range(prompt, prompt + new - 1))], dim=1).double()
    err, bound = (got - exact), (plain - exact)
    rel = lambda e: (e.norm(dim=-1) / exact.norm(dim=-1))
    print(f"\n  B={B} d={d} layers={layers}: relative error {rel(err).mean():.2e} (worst {rel(err).max():.2e}), "
          f"torch's {rel(bound).mean():.2e} ({rel(bound).max():.2e})")
    for part in (slice(0, prompt), slice(prompt, None)):  # the prompt's kernels and the token's
        assert err[:, part].norm() <= bound[:, part].norm()
    assert rel(err).max() <= 1.25 * rel(bound).max()  # the largest of as many draws of about one size
    last = slice(prompt - 1, None)
    chosen, best = tokens[:, prompt:], exact[:, last].argmax(-1)
    assert torch.equal(chosen, got[:, last].argmax(-1))  # generate chose what these logits say
    gap = (exact[:, last].gather(-1, best.unsqueeze(-1)) - exact[:, last].gather(-1, chosen.unsqueeze(-1))).squeeze(-1)
    assert (gap <= 2 * bound[:, last].abs().amax(-1)).all() and (gap[chosen == best] == 0).all()


def small(seed=0, layers=3, d=128, vocab=512):
    w = model_weights(d, layers, vocab, seed=seed)
    return w, decoder(w, layers)


def prompts(n, B=3, P=7, vocab=512, seed=0):
    g = torch.Generator().manual_seed(seed)
    return [torch.randint(0, vocab, (B, P), generator=g).cuda() for _ in range(n)]


def test_a_kept_step_serves_later_calls():
    """A second prompt, another batch, other lengths and a sampled call in between, on one decoder and on fresh ones."""
    w, dec = small()
    fresh = lambda ids, new: decoder(w, 3).generate(ids, new, use_graph=False)
    for ids, new in ((prompts(1)[0], 9), (prompts(1, seed=1)[0], 9), (prompts(1, B=5, seed=2)[0], 4), (prompts(1, P=3, seed=3)[0], 20),
                     (prompts(1)[0], 9), (prompts(1)[0], 2), (prompts(1)[0], 1)):
        assert torch.equal(dec.generate(ids, new), fresh(ids, new))
        assert dec.generate(ids, 3, temperature=0.7, top_k=5).shape == (ids.shape[0], ids.shape[1] + 3)
        assert torch.equal(dec.generate(ids, new), fresh(ids, new))


def test_a_kept_step_sees_changed_weights():
    (w, dec), (w2, _) = small(), small(seed=1)
    ids = prompts(1)[0]
    dec.generate(ids, 8)
    kept = dec._slot.graph
    for t, s in ((w[n], w2[n]) for n in w if n.endswith("proj.weight") or ".mlp." in n or n.startswith("embedding")):
        t.copy_(s)  # in place: the graph reads them where they are
    want = decoder(w, 3).generate(ids, 8, use_graph=False)
    assert torch.equal(dec.generate(ids, 8), want) and dec._slot.graph is kept
    for layer in dec.layers:  # replaced: a step of its own
        layer.conv_w, layer.skip = layer.conv_w * 0.5, layer.skip * 0.5
    got = dec.generate(ids, 8)
    assert dec._slot.graph is not kept and torch.equal(got, dec.generate(ids, 8, use_graph=False))
    with torch.inference_mode():
        assert torch.equal(dec.generate(ids, 8), got)
    assert torch.equal(dec.generate(ids, 8), got)


def test_threads_generate_side_by_side():
    w, dec = small()
    asks = prompts(8, seed=4)
    want = [decoder(w, 3).generate(ids, 24, use_graph=False) for ids in asks]
    torch.cuda.synchronize()
    got, failed = [None] * len(asks), []

    def work(first):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for i in range(first, len(asks), 2):
                    got[i] = dec.generate(asks[i], 24)
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            failed.append(e)

    threads = [threading.Thread(target=work, args=(n,)) for n in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    assert all(torch.equal(a, b) for a, b in zip(got, want))
