"""The time-parallel form of the scan on one GPU (``time_chunks``): the sequence is cut into chunks that run side
by side from exact start states. Checked against the float64 oracle, not only against the lane-serial kernels."""

import importlib

import numpy as np
import pytest
import torch

import slab_math
from oracle import kla_oracle as O
from test_scan_gpu import INPUTS, REDUCED_SLACK, _oracle, _seeded, ratio, rel_err

pytestmark = pytest.mark.gpu
ops = importlib.import_module("kalman-linear-attention_b200.ops")


def _run(kb, g, chunks, *, prior=False, state=True, dtype=torch.float32):
    dev = "cuda"
    ins = [torch.tensor(g[n], dtype=torch.float32, device=dev) for n in INPUTS]
    ins = [t.to(dtype) if n in ("v", "lambda_v", "k", "q") else t for n, t in zip(INPUTS, ins)]
    ins = [t.requires_grad_(True) for t in ins]
    init, extra = None, []
    if state:
        lam0 = torch.tensor(g["lam0"], dtype=torch.float32, device=dev, requires_grad=True)
        eta0 = torch.tensor(g["eta0"], dtype=torch.float32, device=dev, requires_grad=True)
        init, extra = kb.KLAState(lam0, eta0), [lam0, eta0]
    y, y_var, st = kb.kla_scan_b200(*ins, initial_state=init, decode_from_prior=prior, time_chunks=chunks)
    f32 = lambda n: torch.tensor(g[n], dtype=torch.float32, device=dev)
    loss = (y * f32("dy")).sum() + (y_var * f32("dyvar")).sum()
    if state:
        loss = loss + (st.lam * f32("dlam_fin")).sum() + (st.eta * f32("deta_fin")).sum()
    return y, y_var, st, torch.autograd.grad(loss, ins + extra)


@pytest.fixture(scope="module")
def kb():
    import kla_b200

    return kla_b200


@pytest.mark.parametrize("chunks", [2, 4, 8])
@pytest.mark.parametrize("prior", [False, True])
def test_time_chunks_match_the_oracle(kb, chunks, prior):
    g = _seeded(2, 512, 24, 16, seed=21)
    f, b = _oracle(g, prior=prior)
    launches0 = ops._lib.load().kla_b200_launch_count()
    y, y_var, st, grads = _run(kb, g, chunks, prior=prior)
    torch.cuda.synchronize()
    assert ops._lib.load().kla_b200_launch_count() - launches0 == 6  # aggregate, fold, scan; the same three backwards
    names = ["dv", "dlambda_v", "dk", "dq", "da", "dp", "dlam0", "deta0"]
    rows = {"y": ratio(y, f.y), "y_var": ratio(y_var, f.y_var), "lam_fin": ratio(st.lam, f.lam), "eta_fin": ratio(st.eta, f.eta)}
    rows.update({n: ratio(gr, ref) for n, gr, ref in zip(names, grads, b)})
    print(f"\n  C={chunks} prior={prior}: " + " ".join(f"{n}={r:.2f}" for n, r in rows.items()))
    for n, r in rows.items():
        # the chunk start states pass through one float32 rounding of an exactly folded state, so the elementwise
        # budget is that of the plain kernels; the four reduced gradients keep theirs
        assert r <= (REDUCED_SLACK if n in ("dk", "dq", "da", "dp") else 2.0), (n, r)
    for n, gr, ref in zip(names, grads, b):
        assert rel_err(gr, ref) < 2e-3, (n, rel_err(gr, ref))


def test_time_chunks_agree_with_the_plain_kernels_bf16_and_no_state(kb):
    g = _seeded(3, 384, 40, 16, seed=22, state=False)
    for n in ("v", "lambda_v", "k", "q"):
        g[n] = torch.tensor(g[n]).to(torch.bfloat16).double().numpy()
    y1, yv1, st1, g1 = _run(kb, g, 1, state=False, dtype=torch.bfloat16)
    y4, yv4, st4, g4 = _run(kb, g, 3, state=False, dtype=torch.bfloat16)
    torch.testing.assert_close(y4, y1, rtol=2e-5, atol=2e-6)
    torch.testing.assert_close(yv4, yv1, rtol=2e-5, atol=2e-6)
    torch.testing.assert_close(st4.lam, st1.lam, rtol=2e-5, atol=2e-6)
    torch.testing.assert_close(st4.eta, st1.eta, rtol=2e-5, atol=2e-6)
    for a_, b_, n in zip(g4, g1, INPUTS):
        assert rel_err(a_.float(), b_.double().cpu().numpy()) < (1e-2 if a_.dtype == torch.bfloat16 else 1e-4), n


def test_long_sequence_in_chunks_against_oracle(kb):
    """B=1, T=32768 in 8 chunks of 4096: the aggregates are maps of 4096 steps each.
    State, y and all gradients against the float64 oracle."""
    g = _seeded(1, 32768, 32, 16, seed=23)
    f, b = _oracle(g)
    ins = [g[n] for n in INPUTS]
    b32 = O.scan_bwd(*ins, g["dy"], g["dyvar"], g["lam0"], g["eta0"], g["dlam_fin"], g["deta_fin"], dtype=np.float32)
    y, y_var, st, grads = _run(kb, g, 8)
    _, _, _, grads1 = _run(kb, g, 1)
    names = ["dv", "dlambda_v", "dk", "dq", "da", "dp", "dlam0", "deta0"]
    rows = {"y": ratio(y, f.y), "y_var": ratio(y_var, f.y_var), "lam_fin": ratio(st.lam, f.lam), "eta_fin": ratio(st.eta, f.eta)}
    rows.update({n: ratio(gr, ref) for n, gr, ref in zip(names, grads, b)})
    print("\n  T=32768, |err|/(1e-6 + 1e-5|ref|) against the float64 oracle: 8 chunks / plain kernels / float32 oracle")
    for i, n in enumerate(names):
        print(f"    {n:10s} {rows[n]:8.2f} {ratio(grads1[i], b[i]):8.2f} {ratio(b32[i], b[i]):8.2f}")
    for n, r in rows.items():
        if n in ("da", "dp"):
            # sums over 32768 steps: float32 summation noise grows with the length of the sum; the bound is the
            # reference's own gradient contract (tests/test_backends.py:54) and the noise of the plain kernels
            i = names.index(n)
            assert rel_err(grads[i], b[i]) < 2e-3 and r <= max(REDUCED_SLACK, 2.0 * ratio(grads1[i], b[i])), (n, r)
        else:
            assert r <= (REDUCED_SLACK if n in ("dk", "dq") else 2.0), (n, r)


def test_views_that_cannot_be_chunked_fall_back(kb):
    g = _seeded(2, 256, 16, 16, seed=24, state=False)
    dev = "cuda"
    wide = torch.zeros(2, 300, 16, device=dev)
    wide[:, :256] = torch.tensor(g["v"], dtype=torch.float32, device=dev)
    v = wide[:, :256]  # batch stride 300 rows: not L x the time stride
    rest = [torch.tensor(g[n], dtype=torch.float32, device=dev) for n in INPUTS[1:]]
    with torch.no_grad():
        y4, _, _ = kb.kla_scan_b200(v, *rest, time_chunks=4)
        y1, _, _ = kb.kla_scan_b200(v.contiguous(), *rest, time_chunks=1)
    assert torch.equal(y4, y1)


@pytest.mark.parametrize("prior", [False, True])
@pytest.mark.parametrize("L", [1, 2, 8, 9, 70])
def test_aggregates_keep_the_floor_of_a_squared(kb, L, prior):
    """|a| < 1e-6: a^2 is 1e-12 there, and that is all a chain without process noise keeps of what came before. Held to 1e-5 of the
    float64 restatement's values, chain by chain (a few float32 operations, no cancellation but in b0's sum)."""
    g = _seeded(2, L, 5, 12, seed=27)
    g["a"].reshape(-1)[::2] = np.resize([0.0, 1e-9, -5e-7, 0.9999e-6], 30)
    g["p"].reshape(-1)[::4] = 0.0
    dev = {n: torch.tensor(g[n], dtype=torch.float32, device="cuda") for n in (*INPUTS, "dy", "dyvar", "lam0", "eta0")}
    g = {n: t.double().cpu().numpy() for n, t in dev.items()}
    v, lv, k, q, a, p = (dev[n] for n in INPUTS)
    low = np.broadcast_to(np.abs(g["a"]) < 1e-6, (2, 5, 12))
    fa = ops.slab_aggregate(v, lv, k, a, p).double().cpu().numpy()
    ref = slab_math.forward_aggregate(*[g[n] for n in ("v", "lambda_v", "k", "a", "p")])

    def apply(A, P0, m0):
        x = A[..., 0] + A[..., 1] * P0
        return (A[..., 2] + A[..., 3] * P0) / x, (A[..., 4] + A[..., 5] * P0 + A[..., 6] * m0) / x

    for P0, m0 in ((1.0, 0.0), (1e3, -0.7)):
        for got, want in zip(apply(fa, P0, m0), apply(ref, P0, m0)):
            assert np.all(np.abs(got - want)[low] <= 1e-5 * np.abs(want)[low] + 1e-30)
    aa = ops.slab_aggregate(v, lv, k, a, p, q=q, dy=dev["dy"], dy_var=dev["dyvar"], lam0=dev["lam0"], eta0=dev["eta0"], prior=prior)
    aa = aa.double().cpu().numpy()
    ref = slab_math.adjoint_aggregate(*[g[n] for n in INPUTS], g["dy"], g["dyvar"], g["lam0"], g["eta0"], prior)
    for i in (0, 2, 3, 4, 5, 6):  # (K01 is a difference of two numbers; its share is in b0)
        scale = np.abs(ref[..., i]) if i != 3 else np.abs(ref[..., 3]) + np.abs(ref[..., 0]) + 1e-14
        assert np.all(np.abs(aa[..., i] - ref[..., i])[low] <= 2e-5 * scale[low] + 1e-37), i


def test_gradients_through_the_floor_of_a_squared_cross_a_cut(kb):
    """a = 0, and only the steps behind the cut are read: what the steps in front of it get comes through the floor alone. The uncut
    kernels form it without cancellation: equal to 1e-5. The oracle, in information form, takes it as the difference of two numbers
    of order one: 2.2e-16 of them is 2.2e-4 of 1e-12, so 1e-3."""
    g = _seeded(2, 128, 16, 16, seed=28)
    g["a"][:] = 0.0
    g["dy"][:, :64] = g["dyvar"][:, :64] = 0.0
    _, b = _oracle(g)
    cut, uncut = (_run(kb, g, c)[3] for c in (2, 1))
    for i, want in ((1, b.dlambda_v), (2, b.dk)):
        got, plain, want = cut[i].double().cpu().numpy()[:, 63], uncut[i].double().cpu().numpy()[:, 63], want[:, 63]
        assert 0 < np.abs(want).max() < 1e-9
        assert np.linalg.norm(got - plain) <= 1e-5 * np.linalg.norm(plain) and np.linalg.norm(got - want) <= 1e-3 * np.linalg.norm(want)


@pytest.mark.parametrize("B,L,M,S,dtype,chunks,layer", [
    (2, 256, 40, 16, torch.float32, 4, "sensors"),
    (2, 256, 40, 16, torch.float32, 4, "output"),
    (2, 256, 40, 16, torch.bfloat16, 2, "both"),
    (1, 2401, 41, 5, torch.bfloat16, None, "both"),   # a shorter last chunk, rows that TMA cannot read, dead states
    (3, 2410, 33, 64, torch.float32, None, "both"),  # few channels per CTA
])
@pytest.mark.parametrize("grad", [False, True])
def test_scans_with_the_layers_sensors_and_output_path_in_chunks(kb, B, L, M, S, dtype, chunks, layer, grad):
    """log_variance and epilogue with the time axis cut, against the same call uncut. Both lie within 1 and 2 of
    1e-6 + 1e-5 |ref| of the float64 oracle, so outputs and state agree to 3e-5 of their largest value (times a gate of at
    most 4 here: 1.2e-4), the gradients' sums to 1e-4, and bfloat16 results to one rounding (2^-8) as well."""
    F = torch.nn.functional
    g = torch.Generator().manual_seed(L + M)
    rn = lambda *s: torch.randn(*s, generator=g)
    act = lambda t: t.cuda().to(dtype).requires_grad_(grad)
    f32 = lambda t: t.cuda().requires_grad_(grad)
    ins = [act(rn(B, L, M)), act(rn(B, L, M) if layer != "output" else 1 / F.softplus(rn(B, L, M))),
           act(F.normalize(rn(B, L, S), dim=-1)), act(F.normalize(rn(B, L, S), dim=-1)),
           f32(torch.sigmoid(rn(M, S))), f32(F.softplus(rn(M, S)))]
    init = kb.KLAState(f32(F.softplus(rn(B, M, S)) + 0.5), f32(rn(B, M, S)))
    kw = dict(out_dtype=dtype, initial_state=init)
    leaves = [*ins, *init]
    if layer != "output":
        kw["log_variance"] = (1e-3, 2.0)
    if layer != "sensors":
        epi = dict(z=act(rn(B, L, M)), lambda_skip=f32(rn(M)), gate=act(rn(B, L, M)), gate_activation="silu")
        kw["epilogue"] = epi
        leaves += [epi["z"], epi["lambda_skip"], epi["gate"]]
    ups = [rn(B, L, M).cuda().to(dtype), rn(B, L, M).cuda().to(dtype), rn(B, M, S).cuda(), rn(B, M, S).cuda()]
    assert chunks is not None or ops.pick_time_chunks(B, L, M, S, None, tuple(ins[:2]), grad, True) > 1

    def run(c):
        before = ops._lib.load().kla_b200_launch_count()
        y, y_var, st = kb.kla_scan_b200(*ins, time_chunks=c, **kw)
        assert ops._lib.load().kla_b200_launch_count() - before == (1 if c == 1 else 3)
        assert st.lam.is_contiguous() and st.eta.is_contiguous()  # what an in-place step asks for
        outs = [y, y_var, st.lam, st.eta]
        return outs, torch.autograd.grad(outs, leaves, ups) if grad else []

    (o1, g1), (oc, gc) = run(1), run(chunks)
    for x, y in zip(oc, o1):
        y = y.detach()
        assert rel_err(x.float(), y.double().cpu().numpy()) < 1.2e-4 + (2.0 ** -8 if y.dtype == torch.bfloat16 else 0.0)
    for x, y in zip(gc, g1):
        assert rel_err(x.float(), y.double().cpu().numpy()) < (1e-2 if y.dtype == torch.bfloat16 else 1e-4)


@pytest.mark.parametrize("layer", [False, True])
def test_the_environment_variable_holds_at_any_length(kb, monkeypatch, layer):
    g = _seeded(2, 256, 16, 16, seed=25, state=False)
    ins = [torch.tensor(g[n], dtype=torch.float32, device="cuda") for n in INPUTS]
    kw = dict(epilogue=dict(z=ins[0], lambda_skip=ins[4][:, 0].contiguous())) if layer else {}

    def run():
        before = ops._lib.load().kla_b200_launch_count()
        y = kb.kla_scan_b200(*ins, **kw)[0]
        return y, ops._lib.load().kla_b200_launch_count() - before

    y1, n1 = run()
    monkeypatch.setenv("KLA_B200_TIME_CHUNKS", "4")
    y4, n4 = run()
    assert (n1, n4) == (1, 3)
    torch.testing.assert_close(y4, y1, rtol=2e-5, atol=2e-6)
