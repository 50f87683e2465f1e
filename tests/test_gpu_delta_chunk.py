"""The chunked delta-rule kernels (16 steps at a time on the tensor cores) against the float64 oracle
where they can go wrong: lengths around one and two chunks and around the ring of prepared chunks, a
carried state, both element types, dense and time-major rows."""
import math

import pytest
import torch

import srwm_oracle as orc
from conftest import delta_inputs

pytestmark = pytest.mark.gpu
CHUNK_IDS = {16: (2, (2, 3)), 32: (1, (1,)), 64: (1, (1,))}     # head size -> forward id, backward ids


@pytest.mark.parametrize("dtype,time_major", [(torch.float32, False), (torch.bfloat16, False), (torch.float32, True)])
@pytest.mark.parametrize("E", [16, 32, 64])
@pytest.mark.parametrize("L", [1, 15, 16, 17, 31, 32, 33, 49, 81])
def test_chunk_kernels(E, L, dtype, time_major):
    import srwm_b200 as sb
    d = torch.device("cuda", 0)
    Q, K, V, B, W0, go = delta_inputs(2, 3, L, E, 7 + L, "rand")
    Q, K, V, B, go = (t.to(dtype).float() for t in (Q, K, V, B, go))
    f = orc.delta_forward_explicit(*(t.double() for t in (Q, K, V, B, W0)))
    r = orc.delta_backward_explicit(*(t.double() for t in (Q, K, V, B)), f["v_old"], f["v_insert"], go.double(), f["W"])

    def put(t):
        t = t.to(d, dtype)
        return t.permute(2, 0, 1, 3).contiguous().permute(1, 2, 0, 3) if time_major else t

    dev = [put(t) for t in (Q, K, V, B)]
    tol = 8e-3 if dtype == torch.bfloat16 else 5e-6
    fwd, bwds = CHUNK_IDS[E]
    W = W0.to(d).clone()
    out, saved = sb.delta_forward(*dev, W, variant=fwd)
    assert orc.rel_max(out.float().cpu(), f["out"]) < tol
    for a, b in zip((*saved, W), (f["v_old"], f["v_insert"], f["W"])):
        assert orc.rel_max(a.cpu(), b) < 5e-6
    WL = W.clone()
    for v in bwds:
        W.copy_(WL)
        g = sb.delta_backward(*dev, saved, put(go), W, want_grad_W0=True, variant=v)
        for a, b in zip(g[:4], r[:4]):
            assert orc.rel_max(a.float().cpu(), b) < tol
        assert orc.rel_max(g[4].cpu(), r[5]) < 5e-6
        assert float((W.cpu() - W0).abs().max()) < 5e-6
    W.copy_(W0)
    out2, none = sb.delta_forward(*dev, W, save=False, variant=fwd)
    assert none is None and torch.equal(out2, out) and torch.equal(W, WL)


@pytest.mark.parametrize("E,L,dtype", [(64, 130, torch.bfloat16), (64, 257, torch.bfloat16), (32, 130, torch.bfloat16),
                                       (64, 130, torch.float32), (64, 257, torch.float32)])
def test_sequences_that_share_a_multiprocessor(E, L, dtype):
    """More sequences than are resident at once, several waves of prepared chunks each: all of them alike, to the bit, and equal to
    the oracle (tolerance: one rounding of a bf16 result; fp32 sums, ten times what a step-by-step fp32 run on the CPU is off by)."""
    import srwm_b200 as sb
    n = 700
    one = [t.to(dtype).float() if i != 4 else t for i, t in enumerate(delta_inputs(1, 1, L, E, L, "rand"))]
    Q, K, V, B, W0, go = one
    f = orc.delta_forward_explicit(*(t.double() for t in (Q, K, V, B, W0)))
    r = orc.delta_backward_explicit(*(t.double() for t in (Q, K, V, B)), f["v_old"], f["v_insert"], go.double(), f["W"])
    rep = [t.cuda().expand(n, -1, -1, -1).contiguous() for t in one]
    dev, W, g_out = [t.to(dtype) for t in rep[:4]], rep[4], rep[5].to(dtype)
    _, saved = sb.delta_forward(*dev, W)
    g = sb.delta_backward(*dev, saved, g_out, W, want_grad_W0=True)
    tol = 8e-3 if dtype == torch.bfloat16 else 5e-6
    for a, want, t in zip((*g, W), (*r[:4], r[5], W0.double()), (tol,) * 4 + (5e-6,) * 2):
        assert torch.equal(a, a[:1].expand_as(a))
        assert orc.rel_max(a[:1].float().cpu(), want) < t


def _packed_oracle(x, W0, go, eps):
    """Raw rows [q | k | v | b] -> out, v_old, v_insert, final state, gradient of the rows, first state again, its gradient; float64.
    (elu + 1 value by value: with torch's fp32 exp on the host a reference was off by 1e-5 in one run, in the first 1813 of 3626
    values, which are one thread's share, while the kernel's results were right.)"""
    E = W0.shape[-1]
    a = x.double().apply_(lambda v: v + 1.0 if v > 0.0 else math.exp(v))
    Sq, Sk = a[..., :E].sum(-1, True) + eps, a[..., E:2 * E].sum(-1, True) + eps
    q, k, v, b = a[..., :E] / Sq, a[..., E:2 * E] / Sk, x[..., 2 * E:3 * E].double(), x[..., 3 * E:].double().sigmoid()
    f = orc.delta_forward_explicit(q, k, v, b, W0.double())
    gq, gk, gv, gb, W0_again, gW0 = orc.delta_backward_explicit(q, k, v, b, f["v_old"], f["v_insert"], go.double(), f["W"])
    gq = (gq - (gq * q).sum(-1, True)) / Sq * (q * Sq).clamp(max=1)
    gk = (gk - (gk * k).sum(-1, True)) / Sk * (k * Sk).clamp(max=1)
    return f["out"], f["v_old"], f["v_insert"], f["W"], torch.cat([gq, gk, gv, gb * b * (1 - b)], -1), W0_again, gW0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("per_sm,more", [(1, 1), (2, 0), (2, 1), (4, 100)])
@pytest.mark.parametrize("E", [64, 32])
def test_packed_sequences_that_share_a_multiprocessor(E, per_sm, more, dtype):
    """Packed rows at odd offsets, sequences around the lines between the backward's kernels, many rounds of the ring of chunks: all of
    them alike, to the bit, and equal to the oracle (tolerances as above; the rows' own gradients go through a difference of sums of 64)."""
    from srwm_b200.layer_ops import delta_packed_backward, delta_packed_forward
    L, eps = 130, 1e-5
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    g = torch.Generator().manual_seed(E + n)
    x, go = (torch.randn(1, 1, L, w, generator=g).to(dtype) for w in (3 * E + 1, E))
    W0 = 0.1 * torch.randn(1, 1, E, E, generator=g)
    out_o, vo, vi, WL, gx_o, W_o, gW_o = _packed_oracle(x.float(), W0, go.float(), eps)
    rep = lambda t: t.cuda().permute(2, 0, 1, 3).expand(-1, -1, n, -1).contiguous().permute(1, 2, 0, 3)   # [1, n, L, w], time-major
    X, GO, W = rep(x), rep(go), W0.cuda().expand(1, n, E, E).contiguous()
    out, saved = delta_packed_forward(X, W, eps)
    tol = 8e-3 if dtype == torch.bfloat16 else 5e-6
    for a, want, t in zip((out, *saved, W), (out_o, vo, vi, WL), (tol,) + (5e-6,) * 3):
        assert torch.equal(a, a[:, :1].expand_as(a))
        assert orc.rel_max(a[:, :1].float().cpu(), want) < t
    gx, gW0 = delta_packed_backward(X, saved, GO, W, eps, want_grad_W0=True)
    for a, want, t in zip((gx, W, gW0), (gx_o, W_o, gW_o), (max(tol, 1e-5), 5e-6, 5e-6)):
        assert torch.equal(a, a[:, :1].expand_as(a))
        assert orc.rel_max(a[:, :1].float().cpu(), want) < t


def _same(got, want, tol):
    """Infinities and NaN at the same places, finite values within ``tol`` of the largest."""
    got, want = got.double().cpu(), want.double()
    ok, inf = torch.isfinite(want), float("inf")
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got == inf, want == inf) and torch.equal(got == -inf, want == -inf)
    if ok.any():
        assert float((got - want)[ok].abs().max()) <= tol * max(1e-3, float(want[ok].abs().max()))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E", [16, 32, 64])
@pytest.mark.parametrize("where", ["q", "k", "v", "v of the last step", "W0", "go", "nan"])
def test_infinities_reach_what_they_reach_step_by_step(E, where, dtype):
    """One value in the middle of a chunk: the steps before it and the other columns stay finite, and infinities
    are infinities where the loop has them."""
    import srwm_b200 as sb
    L, inf = 40, float("inf")
    Q, K, V, B, W0, go = delta_inputs(2, 3, L, E, 7, "rand")
    Q, K, V, B, go = (t.to(dtype).float() for t in (Q, K, V, B, go))
    if where == "W0":
        W0[1, 1, 3, 5] = -inf
    elif where == "nan":
        V[0, 2, 17, 1] = float("nan")
    else:
        {"q": Q, "k": K, "v": V, "go": go}.get(where, V)[1, 1, L - 1 if "last" in where else 21, 5] = inf
    f = orc.delta_forward_explicit(*(t.double() for t in (Q, K, V, B, W0)))
    r = orc.delta_backward_explicit(*(t.double() for t in (Q, K, V, B)), f["v_old"], f["v_insert"], go.double(), f["W"])
    dev = [t.cuda().to(dtype) for t in (Q, K, V, B)]
    tol = 8e-3 if dtype == torch.bfloat16 else 5e-6
    fwd, bwds = CHUNK_IDS[E]
    W = W0.cuda()
    out, saved = sb.delta_forward(*dev, W, variant=fwd)
    _same(out, f["out"], tol)
    for a, b in zip((*saved, W), (f["v_old"], f["v_insert"], f["W"])):
        _same(a, b, 5e-6)
    for v in bwds:
        Wb = W.clone()
        g = sb.delta_backward(*dev, saved, go.cuda().to(dtype), Wb, want_grad_W0=True, variant=v)
        for a, b in zip(g[:4], r[:4]):
            _same(a, b, tol)
        _same(g[4], r[5], 5e-6)
        _same(Wb, r[4], 5e-6)


@pytest.mark.parametrize("E", [16, 32, 64])
@pytest.mark.parametrize("where", ["q = -inf", "k = -inf", "q = inf", "v = inf", "go"])
def test_infinities_in_packed_rows(E, where):
    """Raw rows [q | k | v | b]; -inf in q or k is a zero of elu + 1, which leaves everything finite."""
    from srwm_b200.layer_ops import delta_packed_backward, delta_packed_forward
    N, H, L, eps, inf = 1, 2, 37, 1e-5, float("inf")
    g = torch.Generator().manual_seed(E)
    x, W0, go = (torch.randn(N, H, L, w, generator=g) for w in (3 * E + 1, E, E))
    W0 = 0.1 * torch.randn(N, H, E, E, generator=g)
    if where == "go":
        go[0, 1, 20, 3] = inf
    else:
        x[0, 1, 20, {"q": 1, "k": E + 2, "v": 2 * E + 3}[where[0]]] = -inf if "-" in where else inf
    out_o, vo, vi, WL, gx_o, W0_again, _ = _packed_oracle(x, W0, go, eps)
    W = W0.cuda()
    out, saved = delta_packed_forward(x.cuda(), W, eps)
    _same(out, out_o, 5e-6)
    for s, t in zip((*saved, W), (vo, vi, WL)):
        _same(s, t, 5e-6)
    gx, _ = delta_packed_backward(x.cuda(), saved, go.cuda(), W, eps)
    _same(gx, gx_o, 1e-5)
    _same(W, W0_again, 5e-6)


@pytest.mark.parametrize("E", [16, 32, 64])
def test_the_backward_of_an_empty_sequence_keeps_its_state(E):
    """Nothing is read where there are no rows, whatever the state holds."""
    import srwm_b200 as sb
    rows = lambda w: torch.empty(2, 3, 0, w, device="cuda")
    for bad in (0.25, float("inf"), float("nan")):
        W = torch.full((2, 3, E, E), 0.5, device="cuda")
        W[1, 2, 3, 4] = bad
        want = W.clone()
        for v in CHUNK_IDS[E][1]:
            g = sb.delta_backward(rows(E), rows(E), rows(E), rows(1), (rows(E), rows(E)), rows(E), W, want_grad_W0=True, variant=v)
            assert torch.equal(W.nan_to_num(9.0, 8.0), want.nan_to_num(9.0, 8.0)) and not bool(g[4].any())
