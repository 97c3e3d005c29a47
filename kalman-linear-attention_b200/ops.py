"""Host side of the ``b200`` backend: the reference's backend-callable contract
over the C-ABI library.

The reference dispatches ``kla_scan(..., backend=name)`` to a callable

    fn(v, lambda_v, k, q, a, p, initial_state=None, decode_from_prior=False)
        -> (y [B,L,M], y_var [B,L,M], KLAState(lam, eta) [B,M,S])

looked up in ``kla.ops.kla_ops._BACKENDS`` (src/kla/ops/kla_ops.py:430-442,
486-541). :func:`kla_scan_b200` is such a callable; :func:`kla_step_b200`
mirrors ``kla_step`` (src/kla/ops/kla_ops.py:293-331). Error behaviour follows
the reference's GPU backends (src/kla/ops/cuda_backend.py:239-275): a request
the kernels cannot serve raises ``NotImplementedError`` naming a backend that
can; nothing falls back silently, and there is no CPU or Triton path.
"""

from __future__ import annotations

import os
import sys
from typing import NamedTuple, Optional

import torch
from torch.autograd import forward_ad

from . import _lib
from ._lib import MAX_DSTATE


class KLAState(NamedTuple):
    """Filter state: posterior precision and information vector, each [B, M, S]
    (same fields as the reference's ``KLAState``, src/kla/ops/kla_ops.py:47-51)."""

    lam: torch.Tensor
    eta: torch.Tensor


def init_state(batch: int, d_model: int, d_state: int, device=None, dtype=torch.float32) -> KLAState:
    """Unit prior: precision 1, zero mean (src/kla/ops/kla_ops.py:54-61)."""
    return KLAState(
        lam=torch.ones(batch, d_model, d_state, device=device, dtype=dtype),
        eta=torch.zeros(batch, d_model, d_state, device=device, dtype=dtype),
    )


def _state_cls():
    """The reference's own KLAState when the reference package is loaded, so
    that callers doing isinstance checks or tuple unpacking see what they expect."""
    mod = sys.modules.get("kla.ops.kla_ops")
    return getattr(mod, "KLAState", KLAState) if mod is not None else KLAState


def _unsupported(msg: str) -> NotImplementedError:
    return NotImplementedError(
        f"The b200 KLA backend {msg}. Use backend='torch' (any device) or 'triton' for this case."
    )


_SM100_CACHE: dict = {}


def _require_device(t: torch.Tensor) -> None:
    """The kernels exist for CUDA tensors on an sm_100 device only."""
    if not t.is_cuda:
        raise _unsupported("requires CUDA tensors")
    _require_sm100(t.device)


def _require_sm100(device: torch.device) -> None:
    idx = device.index if device.index is not None else torch.cuda.current_device()
    ok = _SM100_CACHE.get(idx)
    if ok is None:
        ok = torch.cuda.get_device_capability(idx)[0] == 10
        _SM100_CACHE[idx] = ok
    if not ok:
        raise _unsupported("is compiled for sm_100a (B200) only and this device is not one")


def _rowmajor_last(t: torch.Tensor) -> torch.Tensor:
    """The kernels take a batch and a time stride per tensor but need unit stride
    on the last dimension; anything else is copied once."""
    if t.dim() == 3 and (t.shape[-1] <= 1 or t.stride(-1) == 1):
        return t
    return t.contiguous()


_SM_COUNT: dict = {}


def _forward_segments(lib, dev: torch.device, B: int, L: int, M: int, S: int) -> bool:
    """Whether the forward kernel would cut a problem of this shape into segments (``kla_b200_plan_segments``)."""
    idx = dev.index if dev.index is not None else torch.cuda.current_device()
    if idx not in _SM_COUNT:
        _SM_COUNT[idx] = torch.cuda.get_device_properties(idx).multi_processor_count
    lpc = 1
    while 4 * lpc < S:
        lpc *= 2
    per_cta = 128 // lpc  # channels per CTA of the scan kernels
    return lib.kla_b200_plan_segments(B * ((M + per_cta - 1) // per_cta), L, 0, _SM_COUNT[idx], -1, None) > 1


def _launch_fwd(v, lambda_v, k, q, a, p, lam0, eta0, prior: bool, out_dtype, need_ckpt: bool, sensors=None,
                epilogue=None, raw=None):
    """Allocate outputs (and the checkpoint scratch when a backward will follow)
    and enqueue ``kla_b200_scan_fwd`` on the current stream of the inputs' device."""
    # without checkpoints the kernel still hands long lists of sequences from CTA to CTA in segments, given a little
    # working memory
    segments = not need_ckpt and _forward_segments(_lib.load(), v.device, v.shape[0], v.shape[1], v.shape[2], k.shape[2])
    epi = epilogue or {}
    gate = epi.get("gate")
    return _lib.host().scan_fwd(
        v, lambda_v, k, q, a, p, lam0, eta0, prior, out_dtype == torch.bfloat16, need_ckpt, segments, sensors,
        epi.get("z"), epi.get("lambda_skip"), gate, 0 if gate is None else _lib.ACT[epi.get("gate_activation", "silu")],
        *(raw or (None, None)), 1, 0)


def _launch_fwd_chunked(v, lambda_v, k, q, a, p, lam0, eta0, prior: bool, out_dtype, need_ckpt: bool, chunks: int, sensors=None,
                        epilogue=None, raw=None):
    """:func:`_launch_fwd` with the chunks of every sequence running side by side from exact start states, which are
    returned as well."""
    epi = epilogue or {}
    gate = epi.get("gate")
    return _lib.host().scan_fwd_chunked(
        v, lambda_v, k, q, a, p, lam0, eta0, prior, out_dtype == torch.bfloat16, need_ckpt, sensors,
        epi.get("z"), epi.get("lambda_skip"), gate, 0 if gate is None else _lib.ACT[epi.get("gate_activation", "silu")],
        *(raw or (None, None)), chunks, _chunk_len(v.shape[1], chunks))


def _launch_bwd(v, lambda_v, k, q, a, p, lam0, eta0, ckpt, dy, dy_var, dlam_fin, deta_fin,
                prior: bool, out_dtype, sensors=None):
    """Allocate the gradients and enqueue ``kla_b200_scan_bwd``."""
    return _lib.host().scan_bwd(v, lambda_v, k, q, a, p, lam0, eta0, ckpt, dy, dy_var, dlam_fin, deta_fin, prior,
                                out_dtype == torch.bfloat16, sensors, 1, 0)


def slab_aggregate(v, lambda_v, k, a, p, *, q=None, dy=None, dy_var=None, lam0=None, eta0=None,
                   prior: bool = False) -> torch.Tensor:
    """Launch ``kla_b200_slab_aggregate``: one record per lane that describes how a whole time slab acts on
    the filter state (``dy`` None) or on the backward carry (``dy`` given). Returns [B, M, S, 8] float32."""
    return _lib.host().slab_aggregate(v, lambda_v, k, a, p, q, dy, dy_var, lam0, eta0, prior, None, 1, 0)


# CTAs the backward kernel keeps resident on a B200: 148 SMs x 2
_RESIDENT_CTAS = 296
_MIN_CHUNK_STEPS = 64
_LAYER_CHUNKS_FROM = 1600  # steps from which scans with the layer's sensors or output path can be cut (pick_time_chunks)


def _chunkable(t: Optional[torch.Tensor], B: int, L: int) -> bool:
    """[B, L, X] can be read as [B*C, L/C, X] without a copy."""
    return t is None or B == 1 or t.stride(0) == L * t.stride(1)


def _row_bytes(tensors) -> int:
    """Largest power of two, up to 16, that every row of the [B, L, M] tensors starts on. TMA reads rows of 16."""
    n = 16
    for t in tensors:
        e = t.element_size()
        for x in (t.data_ptr(), t.stride(0) * e if t.shape[0] > 1 else 0, t.stride(1) * e if t.shape[1] > 1 else 0):
            while x % n:
                n //= 2
    return n


def pick_time_chunks(B: int, L: int, M: int, S: int, requested: Optional[int] = None, tensors=(), training: bool = False,
                     layer: bool = False) -> int:
    """Number of time chunks for the time-parallel scan. 1 = the plain lane-serial kernels. ``tensors``: the activations,
    for the alignment of their rows; ``training``: a backward follows; ``layer``: the scan also forms the precisions or
    applies the output path.

    The kernels put one CTA on every 32 / 16 / 8 ... channels (d_state 16 / 32 / 64 ...) of every batch element.
    When that grid leaves most of the GPU empty, the sequence is cut into C chunks that run as B*C batch entries;
    building the chunks' start states costs about half of a forward + backward pass on top (B=2 L=4096 M=1024 in 8
    chunks: 0.23 on 0.44 ms), so chunking is only chosen when the plain grid fills less than a third of the resident CTA
    slots; then up to 16 chunks. Chunks keep at least 64 steps and are equally long where the count divides L, else
    a multiple of 16 steps with a shorter last one (:func:`_chunk_len`). ``requested`` (or the environment variable
    KLA_B200_TIME_CHUNKS) overrides the choice; it is lowered to the nearest usable divisor of L."""
    if requested is None and os.environ.get("KLA_B200_TIME_CHUNKS"):
        requested = int(os.environ["KLA_B200_TIME_CHUNKS"])
    lpc = 1
    while 4 * lpc < S:
        lpc *= 2
    mc = 4 * (32 // lpc)
    ctas = B * ((M + mc - 1) // mc)
    if requested is None:
        # Not below 640 steps, where the uncut kernels are done before three launches are (B=1 L=300 M=512: 27 us against
        # 36 to 52 cut, training 163 against 220 to 275). From about 90 CTAs on cutting breaks even, and only for long
        # sequences (96 CTAs: L=900 66 / 234 uncut, 77 / 246 cut; L=2048 143 / 499 and 148 / 491; L=4096 280 / 985 and
        # 273 / 906). Rows that TMA cannot read are staged too slowly by one CTA of a backward: training gains from 640
        # steps on, inference only where they are not even 4-byte aligned and from 900 steps on. At 94 and 96 CTAs (B, M = 3,
        # 1001; 1, 2981; 6, 497; 2, 1473, all within 3 %), forward / training, uncut and cut: float32 L=641 52 / 229 and
        # 68 / 220, L=1537 116 / 523 and 133 / 450, L=1999 151 / 673 and 161 / 548; bfloat16 rows of 8 bytes (M = 1004, 3004,
        # 500, 1476) 52 / 270 and 72 / 241, 117 / 645 and 139 / 510, 151 / 840 and 168 / 628; odd ones 79 / 517 and 98 / 407,
        # 181 / 1780 and 165 / 1140, 234 / 2420 and 210 / 1495.
        if ctas == 0 or 3 * ctas > _RESIDENT_CTAS or L < 640:
            return 1
        if 10 * ctas > 3 * _RESIDENT_CTAS and L < 2048:
            row = _row_bytes(tensors)
            if row == 16 or not (training or (row < 4 and L >= 900)):
                return 1
        # With the layer's sensors and output path inside, the call stands in a layer, whose host takes longer than a short
        # scan: cutting adds launches and has to shorten what the GPU does beyond that. (The lines are those of calls issued one
        # by one; a captured call, which the GPU's times below would cut from 1000 steps on, is not told apart.) Whole prompts of one layer in us,
        # uncut and cut, bfloat16: B=1 d_model=512 L=1000 162 and 170, L=1500 172 and 169, L=2048 215 and 169; training steps
        # between the projections, B=1 M=1024 L=1000 727 and 770, L=2048 775 and 780, L=2400 875 and 765. By the GPU alone
        # (forward / training step, bfloat16): 48 CTAs (B=2 M=768) L=1000 87 / 307 and 72 / 272; 64 CTAs (B=1 M=2048) L=1000
        # 87 / 311 and 83 / 270, L=4096 335 / 1180 and 237 / 750; 80 CTAs (B=1 M=2560) L=1500 127 / 463 and 130 / 418, L=2048
        # 171 / 616 and 158 / 503; 98 CTAs (B=1 M=3136) L=4096 340 / 1221 and 341 / 1101. Above 32
        # states the forward with the output path holds an SM alone, and only a nearly empty GPU has room for chunks: 16
        # CTAs (S=64 B=1 M=128) L=1000 137 / 466 and 89 / 266, 48 CTAs (B=2 M=192) 139 / 470 and 190 / 413, L=4096 540 / 1879
        # and 650 / 1681, 72 CTAs (B=1 M=576) 542 / 1911 and 885 / 2201.
        if layer and lpc >= 16 and (lpc > 16 or ctas > 16):
            return 1
        if layer and L < (2400 if training else _LAYER_CHUNKS_FROM if ctas <= 75 else 2048 if ctas <= 84 else 8000):
            return 1
        # Whole rounds of the resident slots: enough chunks for one, more rounds while chunks are longer than about 256
        # steps, which evens out the last one. Measured on B200, forward / training step in us: B=1 L=1536 M=1536
        # (48 CTAs) 3 chunks 79 / 233, 4 91 / 287, 6 69 / 208, 8 73 / 227, 16 74 / 235, uncut 108 / 380; B=1 L=8192 M=2048
        # (64 CTAs) 4 chunks 431 / 1367, 16 355 / 1154.
        rounds = 1
        while (want := min(16, rounds * _RESIDENT_CTAS // ctas)) < 16 and L > 288 * want:
            rounds += 1
        if L % want:  # equal chunks where a neighbouring count gives them
            want = next((c for c in (want + 1, want - 1) if 1 < c <= 16 and L % c == 0), want)
    else:
        want = max(1, int(requested))
    want = min(want, max(1, L // _MIN_CHUNK_STEPS), max(1, 65535 // max(B, 1)))
    if requested is None:
        while want > 1 and -(-L // _chunk_len(L, want)) != want:  # rounding the length up can leave fewer chunks
            want = -(-L // _chunk_len(L, want))
        return want
    for c in range(want, 0, -1):
        if L % c == 0:
            return c
    return 1


def _chunk_len(L: int, C: int) -> int:
    """Steps per chunk when ``L`` steps are cut into ``C`` chunks."""
    return L // C if L % C == 0 else (-(-L // C) + 15) // 16 * 16


def _as_chunks(t: Optional[torch.Tensor], C: int) -> Optional[torch.Tensor]:
    """View [B, L, X] as [B*C, L/C, X] (same memory)."""
    if t is None or C == 1:
        return t
    B, L, X = t.shape
    if B == 1:
        return t.as_strided((C, L // C, X), (t.stride(1) * (L // C), t.stride(1), t.stride(2)), t.storage_offset())
    return t.as_strided((B * C, L // C, X), (t.stride(1) * (L // C), t.stride(1), t.stride(2)), t.storage_offset())


def _scan_backward(ctx, v, lambda_v, k, q, a, p, lam0, eta0, ckpt, chunk_state, dy, dy_var, dlam_fin, deta_fin):
    """The scan's gradients, cut into chunks where its forward was (``chunk_state``: their start states)."""
    if (dlam_fin is None) != (deta_fin is None):
        zero = torch.zeros((v.shape[0], v.shape[2], k.shape[2]), device=v.device, dtype=torch.float32)
        dlam_fin = zero if dlam_fin is None else dlam_fin
        deta_fin = zero if deta_fin is None else deta_fin
    if dlam_fin is not None:
        dlam_fin, deta_fin = dlam_fin.float().contiguous(), deta_fin.float().contiguous()
    if ctx.chunks > 1:
        return _lib.host().scan_bwd_chunked(
            v, lambda_v, k, q, a, p, *chunk_state, ckpt, dy, dy_var, dlam_fin, deta_fin, ctx.prior,
            ctx.out_dtype == torch.bfloat16, ctx.sensors, ctx.chunks, _chunk_len(v.shape[1], ctx.chunks))
    return _launch_bwd(v, lambda_v, k, q, a, p, lam0, eta0, ckpt, dy, dy_var, dlam_fin, deta_fin, ctx.prior, ctx.out_dtype,
                       ctx.sensors)


class _KLAScanB200(torch.autograd.Function):
    """Forward and exact backward of the fused scan, both as single kernels.

    Inputs are already canonical: v, lambda_v, k, q share one dtype (float32 or
    bfloat16) with unit last stride; a, p float32 contiguous [M, S]; lam0/eta0
    float32 contiguous [B, M, S] or None."""

    @staticmethod
    def forward(ctx, v, lambda_v, k, q, a, p, lam0, eta0, prior: bool, out_dtype: torch.dtype, sensors=None,
                chunks: int = 1):
        need_grad = any(ctx.needs_input_grad[:8])
        ctx.set_materialize_grads(False)  # an output without a gradient costs nothing below
        ctx.chunks = chunks
        if chunks > 1:
            y, y_var, lam_fin, eta_fin, ckpt, lam_in, eta_in = _launch_fwd_chunked(
                v, lambda_v, k, q, a, p, lam0, eta0, prior, out_dtype, need_grad, chunks, sensors)
            ctx.save_for_backward(v, lambda_v, k, q, a, p, lam0, eta0, ckpt, lam_in, eta_in)
        else:
            y, y_var, lam_fin, eta_fin, ckpt = _launch_fwd(
                v, lambda_v, k, q, a, p, lam0, eta0, prior, out_dtype, need_grad, sensors)
            ctx.save_for_backward(v, lambda_v, k, q, a, p, lam0, eta0, ckpt)
        ctx.prior = prior
        ctx.sensors = sensors
        ctx.out_dtype = out_dtype
        return y, y_var, lam_fin, eta_fin

    @staticmethod
    @torch.autograd.function.once_differentiable  # the hand-written gradients have no graph: a double backward raises
    def backward(ctx, dy, dy_var, dlam_fin, deta_fin):
        v, lambda_v, k, q, a, p, lam0, eta0, ckpt, *chunk_state = ctx.saved_tensors
        B, L, M = v.shape
        dev = v.device
        od = ctx.out_dtype

        def grad_in(g):
            if g is None:
                return None
            if g.dtype != od:
                g = g.to(od)
            return _rowmajor_last(g)

        dy = grad_in(dy)
        dy_var = grad_in(dy_var)
        if dy is None:
            dy = torch.zeros((B, L, M), device=dev, dtype=od)
        dv, dlv, dk, dq, da, dp, dlam0, deta0 = _scan_backward(
            ctx, v, lambda_v, k, q, a, p, lam0, eta0, ckpt, chunk_state, dy, dy_var, dlam_fin, deta_fin)
        if k.dtype != torch.float32:
            dk, dq = dk.to(k.dtype), dq.to(k.dtype)
        has_state = lam0 is not None
        return (dv, dlv, dk, dq, da, dp,
                dlam0 if has_state else None, deta0 if has_state else None, None, None, None, None)


class _KLAScanEpilogueB200(torch.autograd.Function):
    """The scan with the layer's output path inside (kla_layer.py:329-338), for training: the forward kernel
    applies skip and gate at its store and also keeps the scan's own y, y_var; the backward runs the path's
    adjoint (one memory-bound kernel) and then the scan's backward kernel."""

    @staticmethod
    def forward(ctx, v, lambda_v, k, q, a, p, lam0, eta0, z, gate, skip, prior, out_dtype, sensors, gate_act, chunks: int = 1):
        ctx.set_materialize_grads(False)
        need_grad = any(ctx.needs_input_grad[:11])
        B, L, M = v.shape
        epi = {}
        skip_flat = None
        if skip is not None:
            skip_flat = skip.detach().float().reshape(-1).contiguous()
            epi.update(z=z, lambda_skip=skip_flat)
        if gate is not None:
            epi.update(gate=gate, gate_activation=gate_act)
        raw = None
        if need_grad and gate is not None:
            raw = (torch.empty((B, L, M), device=v.device, dtype=out_dtype), torch.empty((B, L, M), device=v.device, dtype=out_dtype))
        chunk_state = (None, None)
        if chunks > 1:
            y, y_var, lam_fin, eta_fin, ckpt, *chunk_state = _launch_fwd_chunked(
                v, lambda_v, k, q, a, p, lam0, eta0, prior, out_dtype, need_grad, chunks, sensors, epi, raw)
        else:
            y, y_var, lam_fin, eta_fin, ckpt = _launch_fwd(v, lambda_v, k, q, a, p, lam0, eta0, prior, out_dtype, need_grad,
                                                           sensors, epi, raw)
        ctx.save_for_backward(v, lambda_v, k, q, a, p, lam0, eta0, ckpt, z, gate, skip_flat, *chunk_state, *(raw or ()))
        ctx.chunks = chunks
        ctx.prior, ctx.sensors, ctx.out_dtype, ctx.gate_act = prior, sensors, out_dtype, gate_act
        ctx.skip_shape, ctx.skip_dtype = (None, None) if skip is None else (skip.shape, skip.dtype)
        return y, y_var, lam_fin, eta_fin

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, dout, dout_var, dlam_fin, deta_fin):
        v, lambda_v, k, q, a, p, lam0, eta0, ckpt, z, gate, skip_flat, lam_in, eta_in, *raw = ctx.saved_tensors
        B, L, M = v.shape
        dev, od = v.device, ctx.out_dtype

        def grad_in(g):
            return None if g is None else _rowmajor_last(g if g.dtype == od else g.to(od))

        dout, dout_var = grad_in(dout), grad_in(dout_var)
        if dout is None:
            dout = torch.zeros((B, L, M), device=dev, dtype=od)
        dy, dy_var, dz, dgate, dskip = _lib.host().epilogue_bwd(
            v, od == torch.bfloat16, dout, dout_var, *(raw or (None, None)), z, gate, skip_flat, _lib.ACT[ctx.gate_act])
        dv, dlv, dk, dq, da, dp, dlam0, deta0 = _scan_backward(
            ctx, v, lambda_v, k, q, a, p, lam0, eta0, ckpt, (lam_in, eta_in), dy, dy_var, dlam_fin, deta_fin)
        if k.dtype != torch.float32:
            dk, dq = dk.to(k.dtype), dq.to(k.dtype)
        has_state = lam0 is not None
        return (dv, dlv, dk, dq, da, dp, dlam0 if has_state else None, deta0 if has_state else None,
                dz, dgate, None if dskip is None else dskip.reshape(ctx.skip_shape).to(ctx.skip_dtype), None, None, None, None, None)


def kla_scan_b200(
    v: torch.Tensor,
    lambda_v: torch.Tensor,
    k: torch.Tensor,
    q: torch.Tensor,
    a: torch.Tensor,
    p: torch.Tensor,
    initial_state=None,
    decode_from_prior: bool = False,
    *,
    out_dtype: Optional[torch.dtype] = None,
    log_variance: Optional[tuple] = None,
    epilogue: Optional[dict] = None,
    time_chunks: Optional[int] = None,
):
    """B200 KLA scan. Same call and return contract as the reference's
    ``kla_scan_torch`` (src/kla/ops/kla_ops.py:188-290): returns
    ``(y, y_var, KLAState)``, float32 unless ``out_dtype`` says otherwise.

    float32 inputs are read in place through their strides (the layer hands the
    scan ``torch.split`` views, src/kla/layers/kla_layer.py:205-207); bfloat16
    inputs are read as bfloat16 and widened in registers, where the reference
    widens them with a copy (kla_ops.py:126-137). ``out_dtype=torch.bfloat16``
    (bfloat16 inputs only) also writes y, y_var as bfloat16 -- what the layer
    would cast them to anyway (kla_layer.py:329-330).

    ``log_variance=(obs_var_min, obs_var_max or None)`` fuses the layer's sensor
    prologue (kla_layer.py:224-231): the ``lambda_v`` argument then holds the
    sensor projection's raw log-variance output ``x``, the kernels form
    ``1 / min(softplus(x) + obs_var_min, obs_var_max)`` in float32 on the way in,
    and the gradient returned for that argument is the one with respect to ``x``.

    ``epilogue=dict(z=, lambda_skip=, gate=, gate_activation="silu")`` fuses the
    layer's output path (kla_layer.py:329-338): ``y += lambda_skip * z``
    (``lambda_skip``: one value or one per channel), then ``y *= g``, ``y_var *= g**2``
    with ``g = act(gate)``; either half may be left out. Differentiable with respect
    to ``z``, ``gate`` and ``lambda_skip`` as well: when a gradient is needed the
    forward also keeps the scan's own y, y_var, and the backward runs the path's
    adjoint as one memory-bound kernel before the scan's backward kernel.

    ``time_chunks``: the time-parallel form of the scan. The reference's parallel
    path scans trace-normalised Moebius matrices and affine pairs over time
    (kla_ops.py:76-123, 248, 274-280); here the sequence is cut into C chunks,
    one pass composes each chunk's map on the filter state, a short fold over the
    chunks gives every chunk its exact start state, and the chunks then run
    through the ordinary kernels side by side (the backward does the same with
    the adjoint carry). ``None`` picks C from the shape (:func:`pick_time_chunks`:
    1 unless B*M is too small to fill the GPU), ``1`` switches it off.
    """
    if not epilogue and v.is_cuda:
        lam0, eta0 = initial_state if initial_state is not None else (None, None)
        if _lib.host().canonical(v, lambda_v, k, q, a, p, lam0, eta0) and (
                out_dtype is None or out_dtype == torch.float32 or out_dtype == v.dtype == torch.bfloat16):
            return _run_scan(v, lambda_v, k, q, a, p, lam0, eta0, decode_from_prior, out_dtype or torch.float32,
                             log_variance, time_chunks)
    _require_device(v)
    if a.dim() != 2:
        raise _unsupported("expects a/p of shape [M, S]")
    if v.dim() != 3 or k.dim() != 3:
        raise ValueError("v, lambda_v must be [B, L, M] and k, q [B, L, S]")
    B, L, M = v.shape
    S = k.shape[2]
    if lambda_v.shape != v.shape or q.shape != k.shape or k.shape[:2] != (B, L):
        raise ValueError("shape mismatch between v, lambda_v [B,L,M] and k, q [B,L,S]")
    if tuple(a.shape) != (M, S) or tuple(p.shape) != (M, S):
        raise ValueError(f"a and p must be [M, S] = [{M}, {S}]")
    if S > MAX_DSTATE:
        raise _unsupported(f"supports d_state <= {MAX_DSTATE} (got {S})")
    tensors = (v, lambda_v, k, q, a, p)
    if any(t.dtype == torch.float64 for t in tensors):
        raise _unsupported("runs in float32 only (float64 inputs are for gradcheck on the torch backend)")
    if any(t.device != v.device for t in tensors):
        raise ValueError("all inputs must be on the same device")

    if all(t.dtype == torch.bfloat16 for t in (v, lambda_v, k, q)):
        act = torch.bfloat16
    else:
        act = torch.float32
    if out_dtype is None:
        out_dtype = torch.float32
    if out_dtype not in (torch.float32, torch.bfloat16) or (out_dtype == torch.bfloat16 and act != torch.bfloat16):
        raise _unsupported("writes float32 outputs, or bfloat16 outputs for bfloat16 inputs")
    v, lambda_v, k, q = (_rowmajor_last(t if t.dtype == act else t.to(act)) for t in (v, lambda_v, k, q))
    a = a.float().contiguous()
    p = p.float().contiguous()
    lam0 = eta0 = None
    if initial_state is not None:
        lam0, eta0 = initial_state
        if tuple(lam0.shape) != (B, M, S) or tuple(eta0.shape) != (B, M, S):
            raise ValueError(f"initial_state must hold [B, M, S] = [{B}, {M}, {S}] tensors")
        lam0 = lam0.float().contiguous()
        eta0 = eta0.float().contiguous()

    if epilogue:
        log_variance = _check_log_variance(log_variance)
        epi = dict(epilogue)
        unknown = set(epi) - {"z", "lambda_skip", "gate", "gate_activation"}
        if unknown:
            raise ValueError(f"unknown epilogue keys {sorted(unknown)}")
        if (epi.get("lambda_skip") is None) != (epi.get("z") is None):
            raise ValueError("epilogue needs z and lambda_skip together")
        for name in ("z", "gate"):
            t = epi.get(name)
            if t is not None:
                if tuple(t.shape) != (B, L, M):
                    raise ValueError(f"epilogue {name} must be [B, L, M]")
                epi[name] = _rowmajor_last(t if t.dtype == act else t.to(act))
        skip = epi.get("lambda_skip")
        if skip is not None:
            if skip.numel() not in (1, M):
                raise ValueError("lambda_skip must hold one value or one per channel")
            if skip.device != v.device:
                skip = skip.to(v.device)
        gate_act = epi.get("gate_activation", "silu")
        if gate_act not in ("silu", "gelu", "relu"):
            raise ValueError("gate_activation must be 'silu', 'gelu' or 'relu'")
        training = _wants_grad(v, lambda_v, k, q, a, p, lam0, eta0, epi.get("z"), epi.get("gate"), skip)
        # short prompts are bound by the host: not even the rule is asked for them (3 of 160 us), unless a count is given
        ask = L >= _LAYER_CHUNKS_FROM or time_chunks is not None or os.environ.get("KLA_B200_TIME_CHUNKS")
        chunks = _chunks_of(v, lambda_v, k, q, time_chunks, training, True) if ask else 1
        if not training:
            if skip is not None:
                epi["lambda_skip"] = skip.float().reshape(-1).contiguous()
            if chunks > 1:
                y, y_var, lam_fin, eta_fin, *_ = _launch_fwd_chunked(
                    v, lambda_v, k, q, a, p, lam0, eta0, bool(decode_from_prior), out_dtype, False, chunks, log_variance, epi)
            else:
                y, y_var, lam_fin, eta_fin, _ = _launch_fwd(
                    v, lambda_v, k, q, a, p, lam0, eta0, bool(decode_from_prior), out_dtype, False, log_variance, epi)
            return y, y_var, _state_cls()(lam=lam_fin, eta=eta_fin)
        y, y_var, lam_fin, eta_fin = _KLAScanEpilogueB200.apply(
            v, lambda_v, k, q, a, p, lam0, eta0, epi.get("z"), epi.get("gate"), skip, bool(decode_from_prior),
            out_dtype, log_variance, gate_act, chunks)
        return y, y_var, _state_cls()(lam=lam_fin, eta=eta_fin)
    return _run_scan(v, lambda_v, k, q, a, p, lam0, eta0, decode_from_prior, out_dtype, log_variance, time_chunks)


def _wants_grad(*tensors) -> bool:
    """Whether the call needs the autograd function: for a backward, or to refuse forward-mode tangents, which it has no
    rule for (a plain launch would drop them)."""
    if torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors):
        return True
    return forward_ad._current_level >= 0 and any(t is not None and forward_ad.unpack_dual(t).tangent is not None for t in tensors)


def _check_log_variance(log_variance):
    if log_variance is None:
        return None
    if len(log_variance) != 2 or not log_variance[0] >= 0.0:
        raise ValueError("log_variance must be (obs_var_min >= 0, obs_var_max or None)")
    return float(log_variance[0]), None if log_variance[1] is None else float(log_variance[1])


def _chunks_of(v, lambda_v, k, q, time_chunks, training: bool, layer: bool) -> int:
    """Time chunks of a call with canonical arguments."""
    B, L, M = v.shape
    if L == 0:
        return 1
    chunks = pick_time_chunks(B, L, M, k.shape[2], time_chunks, (v, lambda_v), training, layer)
    if chunks > 1 and time_chunks is not None and not all(_chunkable(t, B, L) for t in (v, lambda_v, k, q)):
        return 1  # an explicit count is taken for sequences that lie back to back
    return chunks


def _run_scan(v, lambda_v, k, q, a, p, lam0, eta0, prior, out_dtype, log_variance, time_chunks):
    """The scan of canonical arguments, without an epilogue."""
    log_variance = _check_log_variance(log_variance)
    training = _wants_grad(v, lambda_v, k, q, a, p, lam0, eta0)
    chunks = _chunks_of(v, lambda_v, k, q, time_chunks, training, log_variance is not None)
    if not training:  # inference: no autograd node, no checkpoints
        if chunks > 1:
            y, y_var, lam_fin, eta_fin, *_ = _launch_fwd_chunked(
                v, lambda_v, k, q, a, p, lam0, eta0, bool(prior), out_dtype, False, chunks, log_variance)
        else:
            y, y_var, lam_fin, eta_fin, _ = _launch_fwd(
                v, lambda_v, k, q, a, p, lam0, eta0, bool(prior), out_dtype, False, log_variance)
        return y, y_var, _state_cls()(lam=lam_fin, eta=eta_fin)
    y, y_var, lam_fin, eta_fin = _KLAScanB200.apply(
        v, lambda_v, k, q, a, p, lam0, eta0, bool(prior), out_dtype, log_variance, chunks)
    return y, y_var, _state_cls()(lam=lam_fin, eta=eta_fin)


def kla_step_b200(
    v: torch.Tensor,
    lambda_v: torch.Tensor,
    k: torch.Tensor,
    q: torch.Tensor,
    a: torch.Tensor,
    p: torch.Tensor,
    state,
    decode_from_prior: bool = False,
    *,
    inplace: bool = False,
):
    """One decode step on the B200: ``kla_step`` of the reference
    (src/kla/ops/kla_ops.py:293-331). v, lambda_v: [B, M]; k, q: [B, S];
    state: (lam, eta) [B, M, S]. Returns ``(y [B,M], y_var [B,M], new_state)``.

    ``inplace=True`` updates the state tensors where they are (they must be
    float32 and contiguous) instead of allocating new ones. When a gradient is
    required the step is run as a length-1 scan, which has a backward. The two
    routes differ where the reference's own ``kla_step`` and ``kla_scan`` differ:
    the step kernel floors ``phi`` at 1e-12 and clamps the variance
    (kla_ops.py:310-312, 323), the scan leaves ``phi`` unfloored (kla_ops.py:238);
    the values agree except for keys that are zero to within 1e-6.
    """
    lam, eta = state
    if v.is_cuda:
        out = _lib.host().step(v, lambda_v, k, q, a, p, lam, eta, bool(decode_from_prior), bool(inplace))
        if out is not None:
            return out[0], out[1], _state_cls()(lam=out[2], eta=out[3])
    _require_device(v)
    if v.dim() != 2 or k.dim() != 2:
        raise ValueError("v, lambda_v must be [B, M] and k, q [B, S]")
    if torch.is_grad_enabled() and any(
        t.requires_grad for t in (v, lambda_v, k, q, a, p, lam, eta)
    ):
        y, y_var, st = kla_scan_b200(
            v.unsqueeze(1), lambda_v.unsqueeze(1), k.unsqueeze(1), q.unsqueeze(1), a, p,
            initial_state=(lam, eta), decode_from_prior=decode_from_prior)
        return y[:, 0], y_var[:, 0], st
    B, M = v.shape
    S = k.shape[1]
    if tuple(a.shape) != (M, S) or tuple(p.shape) != (M, S) or tuple(lam.shape) != (B, M, S):
        raise ValueError("shape mismatch between v [B,M], k [B,S], a/p [M,S] and the state [B,M,S]")
    if S > MAX_DSTATE:
        raise _unsupported(f"supports d_state <= {MAX_DSTATE} (got {S})")
    if any(t.dtype == torch.float64 for t in (v, lambda_v, k, q, a, p, lam, eta)):
        raise _unsupported("runs in float32 only")
    act = torch.bfloat16 if all(t.dtype == torch.bfloat16 for t in (v, lambda_v, k, q)) else torch.float32

    def row(t):
        t = t if t.dtype == act else t.to(act)
        return t if (t.shape[-1] <= 1 or t.stride(-1) == 1) else t.contiguous()

    v, lambda_v, k, q = row(v), row(lambda_v), row(k), row(q)
    a = a.float().contiguous()
    p = p.float().contiguous()
    if inplace:
        if lam.dtype != torch.float32 or not lam.is_contiguous() or eta.dtype != torch.float32 or not eta.is_contiguous():
            raise ValueError("inplace=True needs float32 contiguous state tensors")
    else:
        lam, eta = lam.float().contiguous(), eta.float().contiguous()
    with torch.no_grad():
        out = _lib.host().step(v, lambda_v, k, q, a, p, lam, eta, bool(decode_from_prior), bool(inplace))
    if out is None:
        raise ValueError("v, lambda_v [B, M], k, q [B, S], a, p [M, S] and the state [B, M, S] must agree in shape and device")
    y, y_var, lam, eta = out
    return y, y_var, _state_cls()(lam=lam, eta=eta)
