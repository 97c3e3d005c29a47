"""Shapes that divide into nothing, against the float64 oracle: rows that are not multiples of 16 bytes (or of 4, in
bfloat16), odd channel counts, odd state sizes, sequences cut into chunks of unequal length."""

import importlib
import os
import sys

import numpy as np
import pytest
import torch

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.dirname(HERE))
import kla_b200  # noqa: E402
from oracle import kla_oracle as O  # noqa: E402

ops = importlib.import_module("kalman-linear-attention_b200.ops")



def _rel(got, ref):
    ref = torch.as_tensor(np.asarray(ref), dtype=torch.float64)
    return ((got.detach().double().cpu() - ref).norm() / (ref.norm() + 1e-30)).item()


@pytest.mark.gpu
@pytest.mark.parametrize("B,L,M,S,dtype", [
    (1, 1037, 33, 16, torch.float32),    # 16 chunks of 80 steps, the last one 77 short; odd channels
    (2, 641, 40, 16, torch.float32),     # chunks of 80 steps and one of a single step
    (1, 700, 7, 16, torch.bfloat16),     # 7 channels in bfloat16, the last chunk short
    (2, 129, 1001, 16, torch.float32),   # too short to cut
    (3, 200, 35, 16, torch.bfloat16),    # bfloat16 rows off every 4-byte boundary
    (2, 77, 34, 24, torch.bfloat16),     # even bfloat16 rows, padded states
    (2, 150, 19, 40, torch.float32),     # k, q of wide states, S not a power of two
    (1, 90, 9, 100, torch.float32),
])
def test_ragged_shapes_match_the_oracle(B, L, M, S, dtype):
    g = torch.Generator().manual_seed(B * L + M)
    rn = lambda *s: torch.randn(*s, generator=g)
    F = torch.nn.functional
    ins = [rn(B, L, M), 1 / F.softplus(rn(B, L, M)), F.normalize(rn(B, L, S), dim=-1), F.normalize(rn(B, L, S), dim=-1)]
    ins = [t.to(dtype).float() for t in ins] + [torch.sigmoid(rn(M, S)), F.softplus(rn(M, S))]
    dy, dyv, dlam, deta = rn(B, L, M), rn(B, L, M), rn(B, M, S), rn(B, M, S)
    n = lambda t: t.double().numpy()
    f = O.scan_fwd(*map(n, ins))
    b = O.scan_bwd(*map(n, ins), n(dy), n(dyv), None, None, n(dlam), n(deta))
    dev = [t.to("cuda", dtype if i < 4 else torch.float32).requires_grad_() for i, t in enumerate(ins)]
    y, y_var, st = kla_b200.kla_scan_b200(*dev)
    grads = torch.autograd.grad([y, y_var, st.lam, st.eta], dev, [t.cuda() for t in (dy, dyv, dlam, deta)])
    for name, got, ref in (("y", y, f.y), ("y_var", y_var, f.y_var), ("lam", st.lam, f.lam), ("eta", st.eta, f.eta)):
        assert _rel(got, ref) < 2e-6, name
    for name, got in zip(("dv", "dlambda_v", "dk", "dq", "da", "dp"), grads):
        assert _rel(got, getattr(b, name)) < (2e-5 if got.dtype == torch.float32 else 4e-3), name


def test_chunks_cover_every_length():
    for L in list(range(1, 300)) + [1040, 1501, 4096, 65537]:
        for B, M in ((1, 16), (2, 1000), (1, 3000)):
            c = ops.pick_time_chunks(B, L, M, 16)
            n = ops._chunk_len(L, c)
            assert (c - 1) * n < L <= c * n and (c == 1 or n >= 64), (L, c, n)


def test_chunks_near_one_cta_per_sm_follow_what_tma_can_read():
    """At 89 to 98 CTAs and below 2048 steps a sequence is cut only where its rows are staged without TMA."""
    pick = lambda B, L, M, dtype, training, stride=0, offset=0: ops.pick_time_chunks(
        B, L, M, 16, None, [torch.empty(B * L * (M + stride) + offset, dtype=dtype)[offset:].view(B, L, M + stride)[..., :M]] * 2, training)
    f32, bf16 = torch.float32, torch.bfloat16
    for B, M in ((3, 1024), (1, 3008), (6, 512)):  # rows of 16 bytes in both types
        for dtype in (f32, bf16):
            for L in (640, 1537, 2047):
                assert pick(B, L, M, dtype, True) == pick(B, L, M, dtype, False) == 1
        assert pick(B, 2048, M, f32, True) > 1 and pick(B, 2048, M, f32, False) > 1
    for B, M in ((3, 1004), (1, 3004), (6, 500)):  # in float32 only
        assert pick(B, 1537, M, f32, True) == 1 and pick(B, 1537, M, bf16, True) > 1 and pick(B, 1537, M, bf16, False) == 1
    for B, M in ((3, 1001), (1, 2981), (6, 497)):  # in neither
        assert pick(B, 700, M, f32, True) > 1 and pick(B, 1537, M, f32, False) == 1
        assert pick(B, 700, M, bf16, True) > 1 and pick(B, 700, M, bf16, False) == 1 and pick(B, 1537, M, bf16, False) > 1
    assert pick(3, 1537, 1024, f32, True, stride=2) > 1 and pick(3, 1537, 1024, f32, True, stride=4) == 1  # slices of wider rows
    assert pick(3, 1537, 1024, f32, True, offset=1) > 1 and pick(3, 1537, 1001, f32, True, stride=23) == 1
    assert pick(1, 639, 3000, bf16, True) == 1 and ops.pick_time_chunks(3, 1537, 1024, 16) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("B,L,M,S", [(1, 1, 4, 1), (2, 15, 9, 16), (1, 16, 3, 12), (3, 17, 33, 4), (1, 70, 130, 16), (80, 33, 20, 16)])
def test_raw_scans_around_their_tiles(B, L, M, S):
    """Both tile shapes of the raw scans (the last case has more CTAs than SMs) against a float64 loop and autograd."""
    g = torch.Generator(device="cuda").manual_seed(L)
    rn = lambda *s: torch.rand(*s, generator=g, device="cuda") + 0.2
    ins = [rn(B, L, M, S).requires_grad_() for _ in range(6)]
    lam0 = rn(B, M, S).requires_grad_()
    ref = [t.detach().double().requires_grad_() for t in (*ins, lam0)]
    lam, eta, r_lam, r_eta = ref[6], torch.zeros_like(ref[6]), [], []
    for t in range(L):
        a, b, c, d, al, r = (x[:, t] for x in ref[:6])
        lam, eta = (a * lam + b) / (c * lam + d), al * eta + r
        r_lam.append(lam)
        r_eta.append(eta)
    outs = [kla_b200.mobius_scan_b200(*ins[:4], lam0), kla_b200.affine_scan_b200(*ins[4:])]
    refs = [torch.stack(r_lam, 1), torch.stack(r_eta, 1)]
    w = [rn(B, L, M, S), rn(B, L, M, S)]
    grads = torch.autograd.grad(outs, [*ins, lam0], w)
    r_grads = torch.autograd.grad(refs, ref, [x.double() for x in w])
    for got, want in zip((*outs, *grads), (*refs, *r_grads)):
        torch.testing.assert_close(got.double(), want, rtol=2e-5, atol=2e-5 * want.abs().mean().item())
