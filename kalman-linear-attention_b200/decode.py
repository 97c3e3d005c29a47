"""Token-by-token decode of one KLA layer on the B200 kernels.

The reference layer's decode route (``KLALayer.forward`` with a state and ``L == 1``,
src/kla/layers/kla_layer.py:295-345) is three projections with elementwise work between
them. ``LayerDecoder.step`` runs a small layer's token of up to eight bfloat16 rows, issued outside a graph capture, as one kernel
(``kla_b200_token``), the projections as ``kla_b200_linear`` for up to 32 bfloat16 rows (large
layers of more than 16 rows only outside a graph capture), the first with the step of ``CausalConv1d`` (src/kla/layers/common.py:87-96) inside, and as library
GEMMs around ``kla_b200_conv_step`` otherwise; between the second and the third stands
``kla_b200_step_layer`` (sensor post-processing, the filter step, skip path and gate;
kla_layer.py:199-231, 277-293, 329-338).

A decoder is built from plain tensors and a plain config dict, so it does not need the
reference package at run time; ``LayerDecoder.from_layer`` reads both off a reference
``KLALayer``. All state is updated in place, which makes a step capturable in a CUDA graph.
"""

from __future__ import annotations

import contextlib
import threading

import torch
import torch.nn.functional as F

from . import _lib
from .ops import kla_scan_b200

CONFIG_KEYS = (
    "d_state", "discretization", "zero_process_noise", "clip_value", "obs_var_min", "obs_var_max",
    "value_rank", "qk_norm", "use_conv", "conv_kernel_size", "conv_activation", "use_gating",
    "gating_activation", "use_lambda_skip", "return_variance", "decode_from_prior",
)


def discretize(weights: dict, config: dict):
    """Discrete (a_bar, p_bar), each [M, S]: the reference's ``KLALayer._compute_aq``
    (src/kla/layers/kla_layer.py:164-190) restated on plain tensors."""
    a = -torch.exp(weights["lambda_log"].float())
    p = weights["process_noise"].float()
    if config["zero_process_noise"]:
        p = p + 1e-12
    else:
        p = p.clamp_min(1e-7)
        if config["clip_value"] is not None:
            p = p.clamp_max(config["clip_value"])
    delta = F.softplus(weights["delta"].float()) + 1e-7
    a_bar = torch.exp(delta * a)
    if config["discretization"] == "ou":
        lam_pos = a.abs().clamp_min(1e-8)
        p_bar = (p / (2.0 * lam_pos)) * (-torch.expm1(-2.0 * lam_pos * delta))
    else:
        p_bar = p * delta
    return a_bar.contiguous(), p_bar.contiguous()


def _require_cuda(x: torch.Tensor) -> None:
    if not x.is_cuda:
        raise NotImplementedError("The b200 decode kernels need CUDA tensors; use the reference layer on this device.")


class LayerDecoder:
    # False where other work of the program shares the GPU: a small layer's token, which as one kernel holds every SM and waits for
    # all that another stream has running, then always takes the separate kernels. 8 rows of d_model 1024 call by call, us a token,
    # one kernel / separate: alone 18.5 / 21.9, beside prompts on another stream 55 / 23, beside training 107 / 23.
    whole_gpu = None  # as ModelDecoder.whole_gpu; None is True here

    def __init__(self, weights: dict, config: dict):
        missing = [k for k in CONFIG_KEYS if k not in config]
        if missing:
            raise ValueError(f"decode config lacks {missing}")
        self.w = weights
        self.cfg = dict(config)
        self.M, self.S = weights["delta"].shape
        if self.S > _lib.MAX_DSTATE:
            raise NotImplementedError(f"The b200 decode kernels support d_state <= {_lib.MAX_DSTATE}; use backend='torch'.")
        if config["use_conv"] and config["conv_kernel_size"] > _lib.MAX_CONV_TAPS:
            raise NotImplementedError(f"The b200 conv step supports up to {_lib.MAX_CONV_TAPS} taps; use backend='torch'.")
        self.a_bar, self.p_bar = discretize(weights, config)
        sensor_out = weights["sensor_proj.weight"].shape[0]
        self.w_value = 0 if config["value_rank"] == "conv" else (
            weights["value_expand.weight"].shape[1] if "value_expand.weight" in weights else self.M)
        self.w_var = sensor_out - self.w_value - 2 * self.S
        skip = weights.get("lambda_skip") if config["use_lambda_skip"] else None
        self.skip = None if skip is None else skip.detach().float().reshape(-1).contiguous()
        self.conv_w = None
        if config["use_conv"]:
            self.conv_w = weights["conv.weight"].detach().float().reshape(self.M, -1).contiguous()
            cb = weights.get("conv.bias")
            self.conv_b = None if cb is None else cb.detach().float().contiguous()

    @classmethod
    def from_layer(cls, layer) -> "LayerDecoder":
        """Read weights and config off a reference ``kla.KLALayer``."""
        weights = {k: v.detach() for k, v in layer.state_dict().items()}
        config = {k: getattr(layer.config, k) for k in CONFIG_KEYS}
        return cls(weights, config)

    def to(self, device) -> "LayerDecoder":
        out = LayerDecoder.__new__(LayerDecoder)
        out.__dict__.update(self.__dict__)
        out.w = {k: v.to(device) for k, v in self.w.items()}
        for name in ("a_bar", "p_bar", "skip", "conv_w", "conv_b"):
            t = getattr(self, name, None)
            setattr(out, name, None if t is None else t.to(device))
        return out

    def init_state(self, batch: int, device, dtype=torch.float32):
        """(conv window [B, M, K-1] or None, lam [B, M, S], eta [B, M, S]) -- kla_layer.py:152-160."""
        conv = None
        if self.cfg["use_conv"]:
            conv = torch.zeros(batch, self.M, self.cfg["conv_kernel_size"] - 1, device=device, dtype=dtype)
        lam = torch.ones(batch, self.M, self.S, device=device, dtype=torch.float32)
        return conv, lam, torch.zeros_like(lam)

    def _linear(self, x, name):
        return F.linear(x, self.w[name + ".weight"], self.w.get(name + ".bias"))

    def _sensors(self, z, sens):
        """Split the sensor projection as ``KLALayer._project_sensors`` does (kla_layer.py:199-216), raw."""
        cfg, M, S = self.cfg, self.M, self.S
        o = 0
        if cfg["value_rank"] == "conv":
            v = z
        else:
            v = sens[..., o:o + self.w_value]
            o += self.w_value
            if "value_expand.weight" in self.w:
                v = self._linear(v, "value_expand")
        ls = sens[..., o:o + self.w_var]
        o += self.w_var
        if "var_expand.weight" in self.w:
            ls = self._linear(ls, "var_expand")
        return v, ls, sens[..., o:o + S], sens[..., o + S:o + 2 * S]

    @torch.no_grad()
    def prefill(self, x: torch.Tensor, state=None):
        """A whole prompt: the layer's ``forward(x, state)`` for ``L > 1`` in inference
        (kla_layer.py:295-345). ``x``: [B, L, d_model]. The projections are library GEMMs; the causal
        convolution runs in ``kla_b200_conv_seq``; the scan runs with the sensor prologue and the skip/gate epilogue inside
        (``kla_scan_b200(log_variance=, epilogue=)``). Returns ``(out, state)`` -- or ``((out, out_var),
        state)`` -- with ``state`` ready for ``step``."""
        _require_cuda(x)
        cfg, M = self.cfg, self.M
        B, L, _ = x.shape
        if state is None:
            state = self.init_state(B, x.device, x.dtype)
        conv_state, lam, eta = state
        projected = self._linear(x, "in_proj")
        z, gate = (projected[..., :M], projected[..., M:]) if cfg["use_gating"] else (projected, None)
        if cfg["use_conv"]:
            # the causal convolution over the prompt, in place of cat + transpose + conv1d + activation + transpose
            zc, new_window = _lib.host().conv_seq(z, self.conv_w, self.conv_b, conv_state.to(z.dtype).contiguous(),
                                                  _lib.ACT[cfg["conv_activation"]])  # z: autocast's type, if it is on
            conv_state.copy_(new_window)
            z = zc
        v, ls, k, q = self._sensors(z, self._linear(z, "sensor_proj"))
        clip = cfg["clip_value"]
        if cfg["qk_norm"]:
            k, q = _lib.host().qk_norm(k, q, max(clip or 0.0, 0.0))
        if clip is not None and (clip <= 0 or not cfg["qk_norm"]):
            k, q = k.clamp(-clip, clip), q.clamp(-clip, clip)
        epi = {}
        if self.skip is not None:
            epi.update(z=z, lambda_skip=self.skip)
        if gate is not None:
            epi.update(gate=gate, gate_activation=cfg["gating_activation"])
        y, y_var, st = kla_scan_b200(
            v, ls, k, q, self.a_bar, self.p_bar, initial_state=(lam, eta), decode_from_prior=cfg["decode_from_prior"],
            out_dtype=x.dtype if x.dtype == torch.bfloat16 else None,
            log_variance=(cfg["obs_var_min"], cfg["obs_var_max"]), epilogue=epi or None)
        lam.copy_(st.lam)
        eta.copy_(st.eta)
        y, y_var = y.to(x.dtype), y_var.to(x.dtype)
        out = self._linear(y, "out_proj")
        if cfg["return_variance"]:
            return (out, F.linear(y_var, self.w["out_proj.weight"].pow(2))), state
        return out, state

    def block_step(self, x: torch.Tensor, state, norm_weight: torch.Tensor, norm_eps: float) -> torch.Tensor:
        """``x + step(rms_norm(x), state)``: a block's mixer half for one token (the mean path of a layer that returns
        variances, src/kla/models/sequence_model.py:47-98)."""
        conv_state, lam, eta = state
        return _lib.host().layer_step(self.w, self.cfg, x, conv_state, lam, eta, self.a_bar, self.p_bar, self.skip,
                                      self.conv_w, getattr(self, "conv_b", None), self.w_value, self.w_var, norm_weight,
                                      norm_eps, False)[0]

    def step(self, x: torch.Tensor, state):
        """One token. ``x``: [B, d_model]; ``state``: the tuple of ``init_state``, updated in place.
        Returns ``out`` [B, d_model], or ``(out, out_var)`` when the config returns variances."""
        _require_cuda(x)
        conv_state, lam, eta = state
        out, y_var = _lib.host().layer_step(self.w, self.cfg, x, conv_state, lam, eta, self.a_bar, self.p_bar, self.skip,
                                            self.conv_w, getattr(self, "conv_b", None), self.w_value, self.w_var, None, 0.0,
                                            self.whole_gpu is not False)
        if self.cfg["return_variance"]:
            return out, F.linear(y_var, self.w["out_proj.weight"].pow(2))
        return out


_under_way: dict = {}  # by device: [stream, model, event behind it or None] of models' calls not known to have ended
_under_way_lock = threading.Lock()


@contextlib.contextmanager
def _announced(model, device):
    """Whether a ``generate`` or ``prefill`` of ``model`` has the GPU to itself, as far as models' calls go: none of another model on
    another stream is still being issued or run. (Those of one model share its kept step and follow one another.) Others see this
    call until the GPU is done with it."""
    if torch.cuda.is_current_stream_capturing():
        yield True
        return
    mine = [torch.cuda.current_stream(device), id(model), None]
    with _under_way_lock:
        calls = _under_way.setdefault(mine[0].device_index, [])
        calls[:] = [c for c in calls if c[2] is None or not _lib.host().event_done(c[2].cuda_event)]
        alone = all(c[0] == mine[0] or c[1] == mine[1] for c in calls)
        calls.append(mine)
    try:
        yield alone
        event = torch.cuda.Event()
        event.record(mine[0])
        mine[2] = event
    except BaseException:
        with _under_way_lock:
            calls[:] = [c for c in calls if c is not mine]
        raise


class _TokenGraph:
    """The decode step of a :class:`ModelDecoder` captured once: state, token and logits buffers and the graph that
    advances them by one token."""

    def __init__(self, dec: "ModelDecoder", batch: int, device, dtype, greedy: bool, whole: bool = True):
        self.whole = whole
        self.state = dec.init_state(batch, device, dtype)
        self.token = torch.zeros(batch, device=device, dtype=torch.long)
        self.work = []  # of the kernel that a whole token is, made by its first run here; replays follow one another
        self.done = None  # recorded behind the last use
        self.stream = torch.cuda.current_stream(device)  # whose memory the buffers are
        side = torch.cuda.Stream(device)
        side.wait_stream(torch.cuda.current_stream(device))
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.stream(side):
            self._token(dec, greedy)  # libraries set themselves up outside the capture
            # captured by hand: torch.cuda.graph collects garbage and empties the allocator's cache first, which every
            # allocation after it then pays for; thread-local, so that other threads may go on allocating
            self.graph.capture_begin(capture_error_mode="thread_local")
            try:
                self.logits = self._token(dec, greedy)
            finally:
                self.graph.capture_end()
        torch.cuda.current_stream(device).wait_stream(side)

    def _token(self, dec, greedy):
        logits = dec._token_logits(self.token, self.state, self.work, self.whole)
        if greedy:
            _lib.host().argmax(logits, self.token)
        return logits

    def reset(self):
        """The prior state, ordered behind whatever used the buffers last. They are memory of the stream whose call made the
        step, the kernel's working memory of the side stream that captured it: a stream that uses them says so to the allocator."""
        stream = torch.cuda.current_stream(self.token.device)
        if self.done is not None:
            stream.wait_event(self.done)
        if stream != self.stream:
            for t in (self.token, *(t for layer in self.state for t in layer if t is not None)):
                t.record_stream(stream)
        for t in self.work:  # of the stream it was captured on
            t.record_stream(stream)
        for conv, lam, eta in self.state:
            if conv is not None:
                conv.zero_()
            lam.fill_(1.0)
            eta.zero_()
        return self.state

    def release(self):
        self.done = torch.cuda.Event()
        self.done.record(torch.cuda.current_stream(self.token.device))


class _GraphSlot:
    """One captured decode step kept for the next call with the same batch, types and weights. A call that finds the slot
    taken (another thread generates) captures a step of its own. Copies of a decoder start with an empty slot."""

    def __init__(self):
        self.lock = threading.Lock()
        self.key = self.graph = None

    def __deepcopy__(self, memo):
        return _GraphSlot()

    def __reduce__(self):
        return _GraphSlot, ()


MODEL_KEYS = ("n_layers", "norm_eps", "mlp", "logit_softcap")


class ModelDecoder:
    """Prompt prefill and token-by-token decode of a whole stack of KLA blocks on the B200 kernels: the
    reference's ``SequenceModel.forward`` with a state and ``SequenceModel.generate``
    (src/kla/models/sequence_model.py:150-173, 200-220).

    A block is ``x += mixer(norm(x))`` then ``x += mlp(norm(x))`` (sequence_model.py:47-98). For one token of up to eight
    sequences in bfloat16 all blocks are one kernel (``kla_b200_token``), for up to 16 a block is six: the projections with norm,
    convolution step, gate and residual sum folded in, and the filter step. For up to 32 sequences large projections are library GEMMs. For a prompt the projections are library GEMMs and what stands between them one kernel each.
    That one kernel holds every SM: the tokens of two streams follow one another where separate kernels overlap, and a token waits for
    all that another stream has running. 256 tokens of 12 blocks of d_model 768, 8 rows each, ms, one kernel / separate ones: one
    ``generate`` 82 / 97, two models at once 174 / 112, four 394 / 157, one beside prompts on another stream 475 / 201. A ``generate``
    that finds another model's ``generate`` or ``prefill`` under way on another stream of its device therefore takes the separate
    kernels, with the same results. ``whole_gpu``, set on a decoder, says which: False where other work of the program shares the GPU, True for
    the one kernel at any time.
    One decoded token is a fixed sequence of launches over state that is updated in place, so ``generate`` captures it in
    a CUDA graph, which it keeps for calls with the same batch, types and weights, and replays it: a token then costs no
    host work but one replay, where the reference's loop issues several hundred small launches per token from Python.

    Built from plain tensors (``SequenceModel.state_dict()``) and plain config dicts; ``from_model`` reads them
    off a reference model. The reference package is not needed at run time."""

    whole_gpu = None  # or True, False

    def __init__(self, weights: dict, layer_configs, model_config: dict):
        missing = [k for k in MODEL_KEYS if k not in model_config]
        if missing:
            raise ValueError(f"model config lacks {missing}")
        self.cfg = dict(model_config)
        self.w = weights
        n = self.cfg["n_layers"]
        if len(layer_configs) != n:
            raise ValueError(f"got {len(layer_configs)} layer configs for {n} layers")
        self.layers = []
        for i in range(n):
            pre = f"blocks.{i}.mixer."
            lw = {k[len(pre):]: v for k, v in weights.items() if k.startswith(pre)}
            self.layers.append(LayerDecoder(lw, layer_configs[i]))
        self._slot, self._shared_slot = _GraphSlot(), _GraphSlot()

    @classmethod
    def from_model(cls, model) -> "ModelDecoder":
        """Read weights and configs off a reference ``kla.SequenceModel`` whose mixers are all KLA layers."""
        weights = {k: v.detach() for k, v in model.state_dict().items()}
        layer_configs = [{k: getattr(blk.mixer.config, k) for k in CONFIG_KEYS} for blk in model.blocks]
        model_config = {k: getattr(model.config, k) for k in MODEL_KEYS}
        dec = cls(weights, layer_configs, model_config)
        dev = model.embedding.weight.device
        return dec.to(dev) if dev.type == "cuda" else dec

    def to(self, device) -> "ModelDecoder":
        out = ModelDecoder.__new__(ModelDecoder)
        out.__dict__.update(self.__dict__)
        out.w = {k: v.to(device) for k, v in self.w.items()}
        out.layers = [layer.to(device) for layer in self.layers]
        out._slot, out._shared_slot = _GraphSlot(), _GraphSlot()
        return out

    def init_state(self, batch: int, device, dtype=torch.float32):
        return [layer.init_state(batch, device, dtype) for layer in self.layers]

    def _norm(self, x, name):  # RMSNorm, src/kla/layers/common.py:45-55
        return self._add_norm(x, None, name)[1]

    def _add_norm(self, x, delta, name):
        """``x + delta`` (``x`` itself when ``delta`` is None) and its norm."""
        return _lib.host().add_norm(x, delta, self.w[name + ".weight"], self.cfg["norm_eps"])

    def _mlp(self, i, x):  # src/kla/layers/common.py:99-122
        pre = f"blocks.{i}.mlp."
        if self.cfg["mlp"] == "swiglu":
            h = _lib.host().swiglu(F.linear(x, self.w[pre + "w12.weight"], self.w.get(pre + "w12.bias")))
            return F.linear(h, self.w[pre + "w3.weight"], self.w.get(pre + "w3.bias"))
        return F.linear(F.gelu(F.linear(x, self.w[pre + "w1.weight"], self.w.get(pre + "w1.bias"))),
                        self.w[pre + "w2.weight"], self.w.get(pre + "w2.bias"))

    def _head(self, x, branch):
        return self._cap(F.linear(self._add_norm(x, branch, "norm_f")[1], self.w["lm_head.weight"]))

    def _cap(self, logits):
        cap = self.cfg["logit_softcap"]
        return logits if cap is None else cap * torch.tanh(logits / cap)

    def _step_blocks(self, x, state, work=None, whole=True):
        """One token through the blocks: of up to eight sequences in bfloat16 all of them as one kernel, at sizes where that pays
        (``work``: a list of its working memory where the caller keeps it; ``whole``: it may take the whole GPU); otherwise norm, mixer
        and residual sum of a block are the layer's step with the norm folded into its first projection and the sum into its last, and
        the MLP likewise."""
        _require_cuda(x)
        host, w, eps, mlp = _lib.host(), self.w, self.cfg["norm_eps"], self.cfg["mlp"]
        if whole and mlp in ("swiglu", "none") and x.dtype == torch.bfloat16 and not torch.is_autocast_enabled("cuda"):
            blocks = [(m.w, m.cfg, *st, m.a_bar, m.p_bar, m.skip, m.conv_w, getattr(m, "conv_b", None), m.w_value, m.w_var,
                       w[f"blocks.{i}.mixer_norm.weight"]) for i, (m, st) in enumerate(zip(self.layers, state))]
            mlps = [] if mlp == "none" else [
                (w[f"blocks.{i}.mlp_norm.weight"], w[f"blocks.{i}.mlp.w12.weight"], w.get(f"blocks.{i}.mlp.w12.bias"),
                 w[f"blocks.{i}.mlp.w3.weight"], w.get(f"blocks.{i}.mlp.w3.bias")) for i in range(len(self.layers))]
            y = host.model_token(x, blocks, mlps, eps, work)
            if y is not None:
                return y
        for i, layer in enumerate(self.layers):
            pre = f"blocks.{i}."
            x = layer.block_step(x, state[i], w[pre + "mixer_norm.weight"], eps)
            if mlp == "swiglu":
                m = pre + "mlp."
                x = host.swiglu_step(x, w[pre + "mlp_norm.weight"], eps, w[m + "w12.weight"], w.get(m + "w12.bias"),
                                     w[m + "w3.weight"], w.get(m + "w3.bias"))
            elif mlp != "none":
                x = x + self._mlp(i, self._norm(x, pre + "mlp_norm"))
        return x

    def _prompt_blocks(self, x, state):
        """A prompt through the blocks, each residual sum together with the norm behind it. Returns the sum and the last
        branch, still to be added (``_add_norm`` with the final norm, or of the position that is needed)."""
        _require_cuda(x)
        branch = None
        for i, layer in enumerate(self.layers):
            x, h = self._add_norm(x, branch, f"blocks.{i}.mixer_norm")
            branch = layer.prefill(h, state[i])[0]
            if isinstance(branch, tuple):  # a layer that returns variances: the mean path (sequence_model.py:85-86)
                branch = branch[0]
            if self.cfg["mlp"] != "none":
                x, h = self._add_norm(x, branch, f"blocks.{i}.mlp_norm")
                branch = self._mlp(i, h)
        return x, branch

    @torch.no_grad()
    def prefill(self, input_ids: torch.Tensor, state=None):
        """A prompt: ``input_ids`` [B, L] -> (logits [B, L, vocab], state ready for ``step``)."""
        x = F.embedding(input_ids, self.w["embedding.weight"])
        _require_cuda(x)
        if state is None:
            state = self.init_state(x.shape[0], x.device, x.dtype)
        with _announced(self, x.device):
            return self._head(*self._prompt_blocks(x, state)), state

    @torch.no_grad()
    def step(self, token: torch.Tensor, state):
        """One token per sequence: ``token`` [B] -> logits [B, vocab]; ``state`` is updated in place."""
        return self._token_logits(token, state, whole=self.whole_gpu is not False)

    def _token_logits(self, token, state, work=None, whole=True):
        x = self._step_blocks(F.embedding(token, self.w["embedding.weight"]), state, work, whole)
        return self._cap(_lib.host().project(x, self.w["lm_head.weight"], None, self.w["norm_f.weight"], self.cfg["norm_eps"], None))

    @torch.no_grad()
    def generate(self, input_ids: torch.Tensor, max_new_tokens: int, temperature: float = 0.0, top_k=None,
                 use_graph: bool = True) -> torch.Tensor:
        """``SequenceModel.generate`` (sequence_model.py:200-220): prefill, then one token at a time from the
        recurrent state. ``temperature <= 0`` is greedy. With ``use_graph`` the per-token work of all layers is
        one CUDA graph replay; sampling happens between replays, on the device."""
        x = F.embedding(input_ids, self.w["embedding.weight"])
        _require_cuda(x)
        with _announced(self, x.device) as alone:
            return self._generate(input_ids, x, max_new_tokens, temperature, top_k, use_graph, alone if self.whole_gpu is None else self.whole_gpu)

    def _generate(self, input_ids, x, max_new_tokens, temperature, top_k, use_graph, whole):
        B, P = input_ids.shape
        greedy = temperature <= 0
        whole = whole or x.dtype != torch.bfloat16 or B > _lib.TOKEN_MAX_ROWS  # (tokens that are separate kernels anyway)
        graph_ctx = self._token_graph(B, x.device, x.dtype, greedy, whole) if use_graph and max_new_tokens > 1 else contextlib.nullcontext()
        with graph_ctx as graph:
            state = graph.reset() if graph is not None else self.init_state(B, x.device, x.dtype)
            # the head sees the last position: the prompt's other logits are not needed
            last = (None if t is None else t[:, -1].contiguous() for t in self._prompt_blocks(x, state))
            token = self._sample(self._head(*last), temperature, top_k)
            if max_new_tokens <= 1:
                return torch.cat((input_ids, token), dim=1)
            out = torch.empty(B, P + max_new_tokens, device=x.device, dtype=torch.promote_types(input_ids.dtype, torch.long))
            out[:, :P] = input_ids
            out[:, P] = token[:, 0]
            tok_buf = token[:, 0].clone() if graph is None else graph.token.copy_(token[:, 0])
            for i in range(P + 1, P + max_new_tokens):
                if graph is None:
                    tok_buf.copy_(self._sample(self._token_logits(tok_buf, state, whole=whole), temperature, top_k)[:, 0])
                else:
                    graph.graph.replay()
                    if not greedy:
                        tok_buf.copy_(self._sample(graph.logits, temperature, top_k)[:, 0])
                out[:, i] = tok_buf
        return out

    @contextlib.contextmanager
    def _token_graph(self, batch: int, device, dtype, greedy: bool, whole: bool = True):
        """The captured decode step for this batch: the kept one when it fits and is free, else a new one. Steps that may take
        the whole GPU and others are kept apart."""
        own = [t for name, t in self.w.items() if ".mixer." not in name]
        layers = [t for layer in self.layers
                  for t in (*layer.w.values(), layer.a_bar, layer.p_bar, layer.skip, layer.conv_w, getattr(layer, "conv_b", None))]
        key = (batch, device, dtype, greedy, torch.is_autocast_enabled("cuda"), torch.get_autocast_dtype("cuda"),
               torch.is_inference_mode_enabled(), _lib.host().stamp(own + layers), dict(self.cfg),
               [(dict(layer.cfg), layer.w_value, layer.w_var) for layer in self.layers])
        slot = self._slot if whole else self._shared_slot
        kept = slot.lock.acquire(blocking=False)
        try:
            if kept and slot.key == key:
                graph = slot.graph
            else:
                if kept and slot.graph is not None:
                    slot.graph.done.synchronize()  # its buffers go back to the allocator: nothing may still read them
                    slot.key = slot.graph = None
                graph = _TokenGraph(self, batch, device, dtype, greedy, whole)
                if kept:
                    slot.key, slot.graph = key, graph
            try:
                yield graph
            finally:
                graph.release()
        finally:
            if kept:
                slot.lock.release()

    @staticmethod
    def _sample(logits, temperature, top_k):  # sequence_model.py:222-234
        if temperature <= 0:
            return _lib.host().argmax(logits, torch.empty(logits.shape[:-1], device=logits.device, dtype=torch.long)).unsqueeze(-1)
        logits = logits / temperature
        if top_k is not None:
            kth = torch.topk(logits, top_k, dim=-1).values[..., -1, None]
            logits = logits.masked_fill(logits < kth, float("-inf"))
        return torch.multinomial(torch.softmax(logits.float(), dim=-1), num_samples=1)
