"""A decoded token as one kernel (``kla_b200_token``) against the separate kernels of a token, to the bit: every sum is taken in
the same order and every result rounded in the same places."""

import ctypes
import os
import sys
import threading
from importlib import import_module

import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
import kla_b200  # noqa: E402

pytestmark = pytest.mark.gpu
lib = import_module("kalman-linear-attention_b200._lib")
EPS = 1e-6
BASE = dict(discretization="ou", zero_process_noise=False, clip_value=None, obs_var_min=1e-4, obs_var_max=None, value_rank="full",
            qk_norm=True, use_conv=True, conv_kernel_size=4, conv_activation="silu", use_gating=True, gating_activation="silu",
            use_lambda_skip=True, return_variance=False, decode_from_prior=False)


def stack(d, M, S, layers, hidden, cfg, bias, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s, scale=1.0: torch.randn(*s, generator=g, device="cuda") * scale
    bf = lambda *s: rn(*s, scale=s[-1] ** -0.5).bfloat16()
    cfg = dict(BASE, d_state=S, **cfg)
    w = {"embedding.weight": rn(64, d).bfloat16(), "lm_head.weight": bf(64, d), "norm_f.weight": (1 + rn(d, scale=0.1)).bfloat16()}
    for i in range(layers):
        b, m = f"blocks.{i}.", f"blocks.{i}.mixer."
        v = 0 if cfg["value_rank"] == "conv" else M
        shapes = {"in_proj": ((2 if cfg["use_gating"] else 1) * M, d), "sensor_proj": (v + M + 2 * S, M), "out_proj": (d, M)}
        for n, s in shapes.items():
            w[m + n + ".weight"] = bf(*s)
            if bias:
                w[m + n + ".bias"] = rn(s[0], scale=0.1).bfloat16()
        K = cfg["conv_kernel_size"]
        w.update({m + "conv.weight": rn(M, 1, K, scale=0.5), m + "delta": rn(M, S) - 4, m + "lambda_log": rn(M, S, scale=0.1),
                  m + "process_noise": torch.full((M, S), 0.01, device="cuda"),
                  m + "lambda_skip": rn(M) if bias else torch.tensor(-1.0, device="cuda")})
        if bias:
            w[m + "conv.bias"] = rn(M, scale=0.1)
        w[b + "mixer_norm.weight"] = w[b + "mlp_norm.weight"] = (1 + rn(d, scale=0.1)).bfloat16()
        if hidden:
            w.update({b + "mlp.w12.weight": bf(2 * hidden, d), b + "mlp.w3.weight": bf(d, hidden)})
            if bias:
                w.update({b + "mlp.w12.bias": rn(2 * hidden, scale=0.1).bfloat16(), b + "mlp.w3.bias": rn(d, scale=0.1).bfloat16()})
    model = dict(n_layers=layers, norm_eps=EPS, mlp="swiglu" if hidden else "none", logit_softcap=None)
    return kla_b200.ModelDecoder(w, [cfg] * layers, model)


def same(a, b):
    return all((x is None) == (y is None) and (x is None or torch.equal(x, y)) for x, y in zip(a, b))


def flat(state):
    return [t for layer in state for t in layer]


def launches(f):
    n0 = lib.load().kla_b200_launch_count()
    out = f()
    return out, lib.load().kla_b200_launch_count() - n0


# one row; a group of eight and one more; more rows of W than SMs and fewer; state sizes with and without vector access, within a
# lane, over a whole warp; more columns than a warp holds of x; every option the kernel reads
@pytest.mark.parametrize("B,d,M,S,layers,hidden,cfg,bias", [
    (1, 64, 128, 16, 2, 176, {}, False),
    (8, 768, 1536, 16, 3, 2048, {}, False),
    (7, 136, 272, 12, 2, 360, dict(conv_kernel_size=2, clip_value=0.3, obs_var_max=2.0), True),
    (8, 264, 520, 33, 2, 704, dict(use_gating=False, conv_kernel_size=7, conv_activation="gelu"), True),
    (3, 40, 64, 128, 2, 0, dict(value_rank="conv", decode_from_prior=True, qk_norm=False), True),
    (5, 72, 24, 3, 2, 16, dict(use_conv=False, gating_activation="relu"), False),
    (2, 2048, 4072, 8, 2, 5464, dict(conv_kernel_size=1, use_lambda_skip=False), False),
    (6, 1024, 2080, 64, 2, 2736, {}, True),
    (4, 128, 256, 16, 35, 344, {}, False),  # more layers than one launch takes
])
def test_a_token_of_a_model_is_that_of_the_separate_kernels(B, d, M, S, layers, hidden, cfg, bias):
    dec = stack(d, M, S, layers, hidden, cfg, bias)
    a, b = (dec.init_state(B, "cuda", torch.bfloat16) for _ in range(2))
    for t in range(3):
        x = torch.randn(B, d, generator=torch.Generator(device="cuda").manual_seed(t), device="cuda").bfloat16()
        got, n = launches(lambda: dec._step_blocks(x, a))
        assert n == (layers + 31) // 32
        want = x
        for i, layer in enumerate(dec.layers):
            pre = f"blocks.{i}."
            want = layer.block_step(want, b[i], dec.w[pre + "mixer_norm.weight"], EPS)
            if hidden:
                m = pre + "mlp."
                want = lib.host().swiglu_step(want, dec.w[pre + "mlp_norm.weight"], EPS, dec.w[m + "w12.weight"], dec.w.get(m + "w12.bias"),
                                              dec.w[m + "w3.weight"], dec.w.get(m + "w3.bias"))
        assert torch.equal(got, want) and same(flat(a), flat(b)), t
        assert torch.isfinite(got.float()).all()
    assert lib.device_status() == 0


@pytest.mark.parametrize("B,d,M,S,cfg,n", [(1, 64, 128, 16, {}, 1), (8, 768, 1536, 16, dict(return_variance=True), 1), (7, 40, 96, 20, dict(use_gating=False), 1),
                                           (8, 1024, 2048, 24, {}, 1), (8, 1024, 2048, 25, {}, 4), (1, 1088, 2176, 16, {}, 4)])
def test_a_lone_layers_token_is_that_of_the_separate_kernels(B, d, M, S, cfg, n):
    """Rows do not see one another: those of a batch of 9, the first that takes the separate kernels, are the reference. Strided x.
    Large layers, and a captured token, take the separate kernels too."""
    layer = stack(d, M, S, 1, 0, cfg, True).layers[0]
    more = layer.init_state(9, "cuda", torch.bfloat16)
    few, kept = ([t[:B].clone() for t in more] for _ in range(2))
    xs = torch.randn(3, 9, d + 8, generator=torch.Generator(device="cuda").manual_seed(0), device="cuda").bfloat16()[..., :d]
    wants = []
    for x in xs:
        got, n_few = launches(lambda: layer.step(x[:B], few))
        want, n_more = launches(lambda: layer.step(x, more))
        assert n_few == n and n_more == 4
        if cfg.get("return_variance"):  # the variance's projection is the library's
            assert (got[1].float() - want[1][:B].float()).norm() <= 2 ** -7 * want[1][:B].float().norm()
            got, want = got[0], want[0]
        wants.append(want[:B])
        assert torch.equal(got, want[:B]) and same(few, [s[:B] for s in more])
    graph, x = torch.cuda.CUDAGraph(), xs[0][:B].clone()
    with torch.cuda.graph(graph):
        out, n_graph = launches(lambda: layer.step(x, kept))
    assert n_graph == 4
    for i in range(3):
        x.copy_(xs[i][:B])
        graph.replay()
        assert torch.equal(out[0] if cfg.get("return_variance") else out, wants[i])


@pytest.mark.parametrize("B,d,M,S,hidden,one", [(1, 64, 768, 64, 176, True), (1, 64, 776, 64, 176, False), (2, 64, 776, 64, 176, True),
                                                (8, 64, 592, 64, 0, True), (8, 64, 600, 64, 0, False), (8, 64, 600, 32, 0, True)])
def test_a_captured_token_is_one_kernel_where_that_is_faster(B, d, M, S, hidden, one):
    """Both sides of the rule's lines on 148 SMs (2368 units of 32 lanes): one launch or the separate kernels, the same bits. Call by
    call the host is slower than either, and a token is one kernel."""
    assert torch.cuda.get_device_properties(0).multi_processor_count == 148
    dec = stack(d, M, S, 1, hidden, {}, False)
    x = torch.randn(B, d, device="cuda").bfloat16()
    a, b = (dec.init_state(B, "cuda", torch.bfloat16) for _ in range(2))
    want, n = launches(lambda: dec._step_blocks(x, b))
    assert n == 1
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got, n = launches(lambda: dec._step_blocks(x, a))
    assert (n == 1) == one
    graph.replay()
    assert torch.equal(got, want) and same(flat(a), flat(b))


def test_tokens_on_streams_and_in_graphs_do_not_meet():
    """Eager tokens of one decoder on several streams and threads, and a captured one replayed meanwhile."""
    dec = stack(256, 512, 16, 2, 688, {}, False)
    x = torch.randn(4, 256, device="cuda").bfloat16()
    fresh = lambda: dec.init_state(4, "cuda", torch.bfloat16)
    want, state = [], fresh()
    for _ in range(30):
        want.append(dec._step_blocks(x, state))
    kept, out = fresh(), []
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured, n = launches(lambda: dec._step_blocks(x, kept))
    assert n == 1
    torch.cuda.synchronize()
    got = [None] * 3

    def work(n):
        with torch.cuda.stream(torch.cuda.Stream()):
            mine = fresh()
            got[n] = [dec._step_blocks(x, mine) for _ in range(30)]
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(n,)) for n in range(3)]
    for t in threads:
        t.start()
    for conv, lam, eta in kept:
        conv.zero_(), lam.fill_(1.0), eta.zero_()
    for _ in range(30):
        graph.replay()
        out.append(captured.clone())
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for run in (*got, out):
        assert all(torch.equal(a, b) for a, b in zip(run, want))


def test_a_wait_for_words_that_never_come_runs_out_and_is_reported():
    """One CTA keeps the outputs of one phase to itself: every CTA gives up after the limit, the status names the wait, and the
    next token is right (it does not take what the broken one left for its own)."""
    dec = stack(64, 128, 16, 2, 176, {}, False)
    x = torch.randn(2, 64, device="cuda").bfloat16()
    want = dec._step_blocks(x, dec.init_state(2, "cuda", torch.bfloat16))
    torch.cuda.synchronize()
    L = lib.load()
    try:
        assert L.kla_b200_test_hooks(3_000_000, 2) == 0
        dec._step_blocks(x, dec.init_state(2, "cuda", torch.bfloat16))
        torch.cuda.synchronize()
        status = ctypes.c_int(0)
        assert L.kla_b200_device_status(ctypes.byref(status)) == 0 and status.value == 0x100 | 41
    finally:
        L.kla_b200_test_hooks(0, -1)
    assert torch.equal(dec._step_blocks(x, dec.init_state(2, "cuda", torch.bfloat16)), want) and lib.device_status() == 0


def test_a_captured_tokens_working_memory_is_kept_until_its_replays_are_done():
    """It was allocated on the side stream of the capture and is used on the caller's: a graph that is dropped with its replays
    still to run must not give it to what that side stream allocates next (streams come from a pool of 32)."""
    decode = import_module("kalman-linear-attention_b200.decode")
    dec = stack(64, 128, 16, 2, 176, {}, False)
    graph = decode._TokenGraph(dec, 2, torch.device("cuda", torch.cuda.current_device()), torch.bfloat16, True)
    (work,) = graph.work
    at, size = work.data_ptr(), work.numel()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)  # 0.1 s
    graph.reset()
    graph.graph.replay()
    graph.release()
    still = graph.done
    del graph, work
    taken = []
    for _ in range(40):
        with torch.cuda.stream(torch.cuda.Stream()):
            taken += [torch.empty(size, dtype=torch.uint8, device="cuda") for _ in range(2)]
    assert not still.query()  # the replay has it all to do
    assert all(not t.data_ptr() <= at < t.data_ptr() + size for t in taken)
    torch.cuda.synchronize()


def test_a_generate_beside_another_stream_leaves_it_room():
    """Another model's call on another stream that the GPU is not done with: separate kernels, the same tokens. Not for calls on the
    same stream or of the same model, nor once the other is done or has failed."""
    a, b = (stack(64, 128, 16, 2, 176, {}, False, seed=s) for s in (0, 1))
    ids = torch.arange(12, device="cuda").view(2, 6)
    want = [m.generate(ids, 24) for m in (a, b)]
    own = b._slot.graph
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for busy in (lambda: a.generate(ids, 24), lambda: a.prefill(ids)):
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000_000)  # 0.1 s
            other = busy()
            assert torch.equal(b.generate(ids, 24), want[1]) and b._shared_slot.graph is None  # behind it on its stream
            torch.cuda._sleep(200_000_000)
            other = busy()
        assert torch.equal(a.generate(ids, 24), want[0]) and a._shared_slot.graph is None  # they share a's kept step
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000_000)
            other = busy()
        got = b.generate(ids, 24)
        assert b._shared_slot.graph is not None and not b._shared_slot.graph.whole
        torch.cuda.synchronize()
        assert torch.equal(got, want[1]) and (isinstance(other, tuple) or torch.equal(other, want[0]))
        b._shared_slot.key = b._shared_slot.graph = None
    with torch.cuda.stream(side), pytest.raises(RuntimeError):
        a.generate(ids, 4, temperature=1.0, top_k=1000)  # of 64
    assert torch.equal(b.generate(ids, 24), want[1]) and b._shared_slot.graph is None
    assert b._slot.graph is own
    for whole in (True, False):
        c = stack(64, 128, 16, 2, 176, {}, False)
        c.whole_gpu = whole
        assert torch.equal(c.generate(ids, 24), want[0]) and torch.equal(c.generate(ids, 24, use_graph=False), want[0])
        assert (c._slot.graph is not None) == whole and (c._shared_slot.graph is None) == whole
        assert (launches(lambda: c.step(ids[:, 0], c.init_state(2, "cuda", torch.bfloat16)))[1] < 4) == whole
        layer, x = c.layers[0], torch.randn(2, 64, device="cuda").bfloat16()
        layer.whole_gpu = whole
        assert launches(lambda: layer.step(x, layer.init_state(2, "cuda", torch.bfloat16)))[1] == (1 if whole else 4)
