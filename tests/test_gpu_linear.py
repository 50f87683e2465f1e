"""The layers' fp32 linear maps and layer norms on this library's kernels against float64: sizes around the
edges of the 128 x 128 x 16 tiles and of the 64 or 128 values of k that an accumulator takes, each orientation
of the operands, long sums (split over CTAs), few rows, the residual in the epilogue, and the gradients."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 3e-6      # of the largest result


def _rand(*s, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + 31 * sum(s))
    return torch.randn(*s, device="cuda", generator=g)


def _err(a, b):
    return float((a.double() - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1, 4, 4), (48, 256, 256), (127, 132, 36), (700, 260, 16), (1030, 260, 252),
                                   (1100, 388, 512), (1100, 388, 788), (256, 256, 3200), (64, 1544, 2052), (1000, 64, 8)])
def test_products(M, N, K, ta, tb):
    from srwm_b200 import _lib as L
    from srwm_b200.ops import _stream
    if ta and M % 4:
        M += 4 - M % 4
    A, B, add = _rand(*((K, M) if ta else (M, K))), _rand(*((K, N) if tb else (N, K)), seed=1), _rand(M, N, seed=2)
    ref = (A.double().t() if ta else A.double()) @ (B.double() if tb else B.double().t())
    for with_add in (False, True):
        out = torch.full((M, N), float("nan"), device="cuda")
        a = L.GemmArgs(A.data_ptr(), B.data_ptr(), add.data_ptr() if with_add else None, out.data_ptr(),
                       M if ta else K, N if tb else K, N, N, M, N, K, ta, tb, 0, None, 0)
        need = L.load().srwm_b200_gemm_scratch_bytes(M, N, K)
        scratch = torch.empty(max(need, 16) // 4, device="cuda")
        a.scratch, a.scratch_bytes = scratch.data_ptr(), need
        L.check(L.load().srwm_b200_gemm_f32(C.byref(a), _stream(A)), "gemm")
        assert _err(out, ref + add.double() if with_add else ref) < TOL
    assert L.load().srwm_b200_gemm_timeouts() == 0


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(1029, 772, 64), (1151, 772, 100), (1153, 900, 128), (1281, 772, 260), (1026, 516, 548),
                                   (2303, 1412, 292), (12801, 388, 132)])
def test_pairs_of_tiles(M, N, K, ta, tb):
    """A last tile without its partner, rows in threes and fewer behind the last four, sums that end inside a stage, at an accumulator's
    last one and behind it, and more units than pairs of CTAs.  What lies beside the rows is NaN."""
    from srwm_b200 import _lib as L
    from srwm_b200.ops import _stream
    if ta and tb:
        K += 1
    A, B, add = _rand(M, K), _rand(N, K, seed=1), _rand(M, N, seed=2)
    ref = A.double() @ B.double().t() + add.double()
    lda, ldb = (M + 3) // 4 * 4 if ta else K, N if tb else K
    if ta:
        Am = torch.full((K, lda), float("nan"), device="cuda")
        Am[:, :M] = A.t()
        A = Am
    B = B.t().contiguous() if tb else B
    need = L.load().srwm_b200_gemm_scratch_bytes(M, N, K)
    scratch, out = torch.empty(max(need, 16) // 4, device="cuda"), torch.full((M, N), float("nan"), device="cuda")
    a = L.GemmArgs(A.data_ptr(), B.data_ptr(), add.data_ptr(), out.data_ptr(), lda, ldb, N, N, M, N, K, ta, tb, 0,
                   scratch.data_ptr(), need)
    L.check(L.load().srwm_b200_gemm_f32(C.byref(a), _stream(A)), "gemm")
    assert not L.load().srwm_b200_gemm_few_rows(M, N, K)
    assert _err(out, ref) < TOL
    assert L.load().srwm_b200_gemm_timeouts() == 0


def _same_with_infinities(got, want, tol=TOL):
    """Infinities and NaN at the same places, finite values within ``tol`` of the largest."""
    got, want = got.double().cpu(), want.double().cpu()
    ok = torch.isfinite(want)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got == float("inf"), want == float("inf")) and torch.equal(got == -float("inf"), want == -float("inf"))
    assert float((got - want)[ok].abs().max()) < tol * float(want[ok].abs().max())


@pytest.mark.parametrize("where", ["a", "b", "both", "nan", "add"])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("M,N,K", [(132, 256, 256), (1200, 1032, 132), (1200, 1032, 1300), (260, 132, 3200)])
def test_products_of_infinities(M, N, K, ta, tb, where):
    """Few rows, one drain, several, a sum cut into parts; at the edges of tiles and of the sums."""
    from srwm_b200 import _lib as L
    from srwm_b200.ops import _stream
    inf = float("inf")
    A, B, add = _rand(M, K), _rand(N, K, seed=1), _rand(M, N, seed=2)
    if where in ("a", "both"):
        A[0, 0], A[M - 1, K - 1], A[128, 7], A[128, 8] = inf, -inf, inf, inf
    if where in ("b", "both"):
        B[N - 1, K - 2], B[64, 3] = inf, -inf
        A[5, K - 2] = 0.0                        # 0 * inf
    if where == "nan":
        A[17, K // 2] = float("nan")
    if where == "add":
        add[4, 4], add[M - 1, N - 1] = inf, -inf
    ref = A.double() @ B.double().t() + add.double()
    Am, Bm = (A.t().contiguous() if ta else A), (B.t().contiguous() if tb else B)
    out = torch.empty(M, N, device="cuda")
    need = L.load().srwm_b200_gemm_scratch_bytes(M, N, K)
    scratch = torch.empty(max(need, 16) // 4, device="cuda")
    a = L.GemmArgs(Am.data_ptr(), Bm.data_ptr(), add.data_ptr(), out.data_ptr(), M if ta else K, N if tb else K, N, N,
                   M, N, K, ta, tb, 0, scratch.data_ptr(), need)
    L.check(L.load().srwm_b200_gemm_f32(C.byref(a), _stream(A)), "gemm")
    _same_with_infinities(out, ref)


@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_infinities_with_work_behind_them(ta, tb):
    """Whole tiles that are summed again, all the way to their last value of k, by CTAs that have another unit behind them: nobody's wait
    for those CTAs runs out meanwhile."""
    from srwm_b200 import _lib as L
    from srwm_b200.ops import _stream
    M, N, K = 6652, 264, 8192        # 26 x 3 pairs of tiles on 74 pairs of multiprocessors
    A, B = _rand(M, K), _rand(N, K, seed=1)
    A[:256, K - 2] = float("inf")    # the first three units
    A[300, K - 1], B[200, K - 4] = float("nan"), -float("inf")
    ref = A.double() @ B.double().t()
    Am, Bm = (A.t().contiguous() if ta else A), (B.t().contiguous() if tb else B)
    out = torch.empty(M, N, device="cuda")
    assert L.load().srwm_b200_gemm_scratch_bytes(M, N, K) == 0
    a = L.GemmArgs(Am.data_ptr(), Bm.data_ptr(), None, out.data_ptr(), M if ta else K, N if tb else K, 0, N, M, N, K, ta, tb, 0, None, 0)
    L.check(L.load().srwm_b200_gemm_f32(C.byref(a), _stream(A)), "gemm")
    assert bool(out[:256].isinf().any()) and bool(out[256:].isfinite().any())
    _same_with_infinities(out, ref)
    assert L.load().srwm_b200_gemm_timeouts() == 0


@pytest.mark.parametrize("rows,D", [(1, 4), (7, 132), (300, 256), (9, 512), (6001, 1024)])
def test_layer_norm(rows, D):
    from srwm_b200 import _lib as L
    x, w, b, dy = _rand(rows, D) * 3 + 1, _rand(D, seed=1), _rand(D, seed=2), _rand(rows, D, seed=3)
    leaves = [t.requires_grad_() for t in (x, w, b)]
    y = L.host().layer_norm(*leaves, 1e-5)
    got = torch.autograd.grad(y, leaves, dy)
    ref_leaves = [t.detach().double().requires_grad_() for t in leaves]
    ref = torch.nn.functional.layer_norm(ref_leaves[0], (D,), ref_leaves[1], ref_leaves[2], 1e-5)
    want = torch.autograd.grad(ref, ref_leaves, dy.double())
    assert _err(y.detach(), ref.detach()) < TOL
    for a, r in zip(got, want):
        assert float((a.double() - r).abs().max()) < 4e-6 * max(1.0, float(r.abs().max()))


@pytest.mark.parametrize("lead,N,K", [((3, 5), 64, 32), ((40, 13), 196, 260)])
def test_linear_with_autograd(lead, N, K):
    from srwm_b200 import _lib as L
    x, w, r, dy = _rand(*lead, K), _rand(N, K, seed=1), _rand(*lead, N, seed=2), _rand(*lead, N, seed=3)
    leaves = [t.requires_grad_() for t in (x, w, r)]
    got = torch.autograd.grad(L.host().linear(*leaves), leaves, dy)
    ref_leaves = [t.detach().double().requires_grad_() for t in leaves]
    want = torch.autograd.grad(ref_leaves[2] + ref_leaves[0] @ ref_leaves[1].t(), ref_leaves, dy.double())
    for a, b in zip(got, want):
        assert _err(a, b) < TOL
    no_add = torch.autograd.grad(L.host().linear(x, w, None), (x, w), dy)
    for a, b in zip(no_add, want):
        assert _err(a, b) < TOL
    assert L.host().linear(x.detach().half(), w.detach(), None) is NotImplemented


@pytest.mark.parametrize("rows,N,K", [(1, 4, 4), (48, 512, 256), (50, 20, 132), (3000, 256, 384)])
def test_linear_with_a_bias(rows, N, K):
    from srwm_b200 import _lib as L
    x, w, b = _rand(2, rows, K), _rand(N, K, seed=1), _rand(N, seed=2)
    out = L.host().linear(x, w, b)
    assert _err(out, x.double() @ w.double().t() + b.double()) < TOL
    assert L.host().linear(x, w, b.requires_grad_()) is NotImplemented


@pytest.mark.parametrize("L,B,H,d", [(1, 48, 8, 32), (1, 3, 4, 16), (5, 2, 4, 64)])
def test_layer_steps_without_gradients_equal_those_with(L, B, H, d):
    """One call for the whole layer against the parts (which run where gradients are on)."""
    from srwm_b200.layers import FastFFlayer, FastFFlayerRL, SRlayer
    h = _rand(L, B, H * d)
    state = [0.1 * _rand(B, H, d, w, seed=w) for w in (d, d, d, 4)]
    net = SRlayer(H, d, H * d, 0.0).cuda()
    want, want_state = net(h, state)
    with torch.no_grad():
        got, got_state = net(h, state)
    assert _err(got, want.detach().double()) < TOL
    for a, b in zip(got_state, want_state):
        assert float((a - b).abs().max()) < 1e-5
    W = 0.1 * _rand(B, H, d, d, seed=9)
    net = FastFFlayerRL(H, d, H * d, 0.0).cuda()
    Wa, Wb = W.clone(), W.clone()
    want, _ = net(h, Wa)
    with torch.no_grad():
        got, got_W = net(h, Wb)
    assert _err(got, want.detach().double()) < TOL
    assert float((Wa - Wb).abs().max()) < 1e-5 and torch.equal(got_W, Wb)
    net = FastFFlayer(H, d, H * d, 0.0).cuda()
    with torch.no_grad():
        got = net(h)
    assert _err(got, net(h).detach().double()) < TOL


@pytest.mark.parametrize("T,B,H,d,per_sample", [(1, 3, 8, 32, False), (17, 1, 4, 16, False), (33, 5, 2, 64, False), (9, 3, 4, 16, True)])
def test_unroll_as_one_node_equals_its_parts(T, B, H, d, per_sample):
    """Outputs, final state and every gradient; a hook on the projection makes the layer take its parts."""
    from srwm_b200.layers import SRlayer
    net = SRlayer(H, d, H * d, 0.0).cuda()
    if per_sample:
        for n in ("W_y", "W_q", "W_k", "w_b"):
            setattr(net, n, torch.nn.Parameter(getattr(net, n).detach().repeat(B, 1, 1, 1)))
    done = (torch.arange(T * B, device="cuda").view(T, B) % 7) == 3
    state = [0.1 * _rand(B, H, d, w, seed=w) for w in (d, d, d, 4)]
    gout = _rand(T, B, H * d, seed=5)

    def go():
        h = _rand(T, B, H * d, seed=3).requires_grad_()
        out, st = net.unroll(h, done, state)
        with torch.no_grad():
            out_n, st_n = net.unroll(h, done, state)
        assert torch.equal(out_n, out) and all(torch.equal(a, b) for a, b in zip(st, st_n))
        assert not any(s.requires_grad for s in st)
        return [out, *st, *torch.autograd.grad(out, [h] + list(net.parameters()), gout, allow_unused=True)]
    got = go()
    handle = net.out_linear.register_forward_hook(lambda *a: None)
    want = go()
    handle.remove()
    for a, b in zip(got, want):
        assert (a is None) == (b is None)
        assert a is None or a.shape == b.shape and float((a - b).detach().abs().max()) <= 1e-5 * max(1.0, float(b.detach().abs().max()))


@pytest.mark.parametrize("rows,width", [(1, 64), (48, 512), (3000, 256)])
def test_feed_forward_stack_without_gradients(rows, width):
    """Few rows and many (whose ReLU is a pass of its own), a ReLU behind a product and one that is not."""
    from srwm_b200.layers import _feed_forward
    net = torch.nn.Sequential(torch.nn.LayerNorm(64), torch.nn.ReLU(), torch.nn.Linear(64, width), torch.nn.ReLU(),
                              torch.nn.Linear(width, 64, bias=False)).cuda()
    x = _rand(2, rows, 64)
    want = net.double()(x.double()).detach()
    net.float()
    with torch.no_grad():
        assert _err(_feed_forward(net, x), want) < TOL


@pytest.mark.parametrize("switch,on,off", [("fp32_precision", "tf32", "ieee"), ("allow_tf32", True, False)])
def test_both_tf32_switches_hand_the_products_to_the_library(switch, on, off):
    """... and turn back; the newer one makes the older one's query throw.  In a child process: torch does not let the
    two be mixed."""
    import subprocess
    import sys

    from conftest import ROOT
    code = f"""
import torch, sys
sys.path.insert(0, {ROOT!r} + "/modern-srwm_b200")
from srwm_b200 import _lib as L
from srwm_b200.layers import FastFFlayer
x, w = torch.randn(40, 64, device="cuda"), torch.randn(64, 64, device="cuda")
net, h = FastFFlayer(4, 16, 64, 0.0).cuda(), torch.randn(5, 3, 64, device="cuda")
want = net(h)
m = torch.backends.cuda.matmul
m.{switch} = {on!r}
assert L.host().linear(x, w, None) is NotImplemented
assert float((net(h) - want).abs().max()) < 1e-2
m.{switch} = {off!r}
assert L.host().linear(x, w, None) is not NotImplemented
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def _second(f, leaves, wrt):
    """Gradients of the squares of f's gradients."""
    leaves = [t.detach().clone().requires_grad_() for t in leaves]
    first = torch.autograd.grad(f(*leaves[:-1]), leaves[:-1], leaves[-1], create_graph=True)
    return torch.autograd.grad(sum((t * t).sum() for t in first), [leaves[i] for i in wrt], allow_unused=True)


def test_second_derivatives_equal_the_modules():
    """A gradient penalty: what torch's own linear map and layer norm give."""
    from srwm_b200 import _lib as L
    F = torch.nn.functional
    x, w, r, dy = _rand(40, 13, 260), _rand(196, 260, seed=1), _rand(40, 13, 196, seed=2), _rand(40, 13, 196, seed=3)
    for with_r in (True, False):
        args, wrt = ((x, w, r, dy), (0, 1, 3)) if with_r else ((x, w, dy), (0, 1, 2))
        got = _second(lambda *a: L.host().linear(*a, *([] if with_r else [None])), args, wrt)
        want = _second(lambda x, w, r=0.0: r + F.linear(x, w), [t.double() for t in args], wrt)
        for a, b in zip(got, want):
            assert _err(a, b) < 1e-5
    x, w, b, dy = _rand(40, 132), _rand(132, seed=1), _rand(132, seed=2), _rand(40, 132, seed=3)
    got = _second(lambda *a: L.host().layer_norm(*a, 1e-5), (x, w, b, dy), (0, 1, 3))
    want = _second(lambda x, w, b: F.layer_norm(x, (132,), w, b, 1e-5), [t.double() for t in (x, w, b, dy)], (0, 1, 3))
    for a, b in zip(got, want):
        assert _err(a, b) < 1e-5


def test_second_derivatives_of_the_unroll_equal_its_parts():
    from srwm_b200.layers import SRlayer
    T, B, H, d = 5, 3, 4, 16
    torch.manual_seed(0)
    net = SRlayer(H, d, H * d, 0.0).cuda()
    done = (torch.arange(T * B, device="cuda").view(T, B) % 7) == 3
    state = [0.1 * _rand(B, H, d, w, seed=w) for w in (d, d, d, 4)]

    def go():
        h, gout = _rand(T, B, H * d).requires_grad_(), _rand(T, B, H * d, seed=5).requires_grad_()
        leaves = [h, net.W_y, net.out_linear.weight]
        first = torch.autograd.grad(net.unroll(h, done, state)[0], leaves, gout, create_graph=True)
        return (*first, *torch.autograd.grad(sum((t * t).sum() for t in first), leaves + [gout], allow_unused=True))
    got = go()
    handle = net.out_linear.register_forward_hook(lambda *a: None)
    want = go()
    handle.remove()
    assert [t is None for t in got] == [t is None for t in want] and got[3] is not None and got[4] is not None
    for a, b in zip(got, want):
        assert a is None or float((a - b).detach().abs().max()) <= 1e-5 * float(b.detach().abs().max())


@pytest.mark.parametrize("grad", [False, True])
def test_an_unroll_without_done_is_refused(grad):
    from srwm_b200.layers import SRlayer
    net = SRlayer(4, 16, 64, 0.0).cuda()
    state = [0.1 * _rand(3, 4, 16, w, seed=w) for w in (16, 16, 16, 4)]
    with torch.set_grad_enabled(grad), pytest.raises(AttributeError):
        net.unroll(_rand(5, 3, 64), None, state)


def _odd(t):
    """The same values at an address or with strides that no kernel takes as they are: off by one element, or the first
    dimension innermost with gaps."""
    if t.dim() == 1:
        return t.new_empty(t.numel() + 1)[1:].copy_(t)
    strides, run = [], 2
    for n in t.shape:
        strides.append(run)
        run *= n
    return torch.empty_strided(t.shape, strides, dtype=t.dtype, device=t.device).copy_(t)


@pytest.mark.parametrize("kind", ["unroll", "layer", "stateful", "delta", "delta layer", "operator"])
@pytest.mark.parametrize("hooks", ["odd strides", "on the CPU"])
def test_saved_tensor_hooks(kind, hooks):
    """What the hooks give back may lie in memory in another way than what was saved."""
    import srwm_b200 as sb
    from srwm_b200.layers import FastFFlayer, SRlayer, SRWMlayer
    T, B, H, d = 19, 3, 4, 16
    torch.manual_seed(0)
    h = _rand(T, B, H * d).requires_grad_()
    state = [(0.1 * _rand(B, H, d, w, seed=w)).requires_grad_(kind != "unroll") for w in (d, d, d, 4)]
    done = (torch.arange(T * B, device="cuda").view(T, B) % 7) == 3
    leaves = [h]
    if kind == "unroll":
        net = SRlayer(H, d, H * d, 0.0).cuda()
        f = lambda: net.unroll(h, done, state)[0]
    elif kind == "layer":
        net = SRWMlayer(H, d, H * d, 0.0, use_input_softmax=True).cuda()
        f = lambda: net(h)
    elif kind == "stateful":
        net = SRWMlayer(H, d, H * d, 0.0, stateful=True).cuda()
        leaves = leaves + state
        f = lambda: torch.cat([t.flatten() for t in (lambda o, s: (o, *s))(*net(h, state, True))])
    elif kind == "delta layer":
        net = FastFFlayer(H, d, H * d, 0.0).cuda()
        f = lambda: net(h)
    else:
        net = None
        x = torch.softmax(_rand(B, H, T, d), -1).requires_grad_()
        W = [_rand(B, H, d, w, seed=w).mul(0.2).requires_grad_() for w in (d, d, d, 4)]
        beta = torch.sigmoid(_rand(B, H, T, 1)).requires_grad_()
        leaves = [x, beta] if kind == "delta" else [x] + W
        f = ((lambda: sb.fast_weight_delta(x, x * 1.0, x * 2.0, beta, torch.zeros(B, H, d, d, device="cuda"))) if kind == "delta"
             else lambda: sb.self_ref_v0(x, *[w.clone() for w in W]))
    leaves = leaves + (list(net.parameters()) if net is not None else [])
    want = torch.autograd.grad(f().square().sum(), leaves, allow_unused=True)
    ctx = (torch.autograd.graph.save_on_cpu() if hooks == "on the CPU"
           else torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: _odd(t.detach())))
    with ctx:
        out = f().square().sum()
    got = torch.autograd.grad(out, leaves, allow_unused=True)
    for a, b in zip(got, want):
        assert (a is None) == (b is None)
        assert a is None or float((a - b).abs().max()) <= 1e-5 * max(1.0, float(b.abs().max()))


def test_what_asks_for_the_modules_gets_them():
    """A forward of the instance's own, a backward hook on the idle dropout, hooks of a whole stack, forward-mode AD."""
    import torch.autograd.forward_ad as fw

    from srwm_b200 import _lib as L
    from srwm_b200.layers import FastFFlayer, SRlayer, _feed_forward
    net = SRlayer(4, 16, 64, 0.0).cuda()
    state = [0.1 * _rand(3, 4, 16, w, seed=w) for w in (16, 16, 16, 4)]
    h, done, calls = _rand(5, 3, 64), torch.zeros(5, 3, dtype=torch.bool, device="cuda"), []
    own = net.out_linear.forward
    net.out_linear.forward = lambda x: (calls.append("forward"), own(x))[1]
    net.unroll(h, done, state)
    with torch.no_grad():
        net(h[:1], state)
    assert calls == ["forward"] * 2
    del net.out_linear.forward, calls[:]
    net.drop.register_full_backward_hook(lambda *a: calls.append("drop"))
    net.unroll(h, done, state)[0].sum().backward()
    assert calls == ["drop"]
    stack = torch.nn.Sequential(torch.nn.LayerNorm(64), torch.nn.Linear(64, 64)).cuda()
    handle = torch.nn.modules.module.register_module_forward_hook(lambda m, *a: calls.append(type(m).__name__))
    del calls[:]
    with torch.no_grad():
        _feed_forward(stack, h)
    handle.remove()
    assert calls == ["LayerNorm", "Linear", "Sequential"]
    x, w = _rand(40, 64), _rand(64, 64, seed=1)
    layer = FastFFlayer(4, 16, 64, 0.0).cuda().requires_grad_(False)
    with fw.dual_level():
        dual = fw.make_dual(x, torch.ones_like(x))
        assert L.host().linear(dual, w, None) is NotImplemented and L.host().layer_norm(dual, w[0], w[1], 1e-5) is NotImplemented
        for grad in (True, False):
            with torch.set_grad_enabled(grad), pytest.raises(Exception, match="forward"):
                fw.unpack_dual(layer(fw.make_dual(h, h)))


def test_the_first_product_of_a_process_may_be_captured():
    """The word in host memory that a kernel sets when it gives up is then taken during the capture."""
    import subprocess
    import sys

    from conftest import ROOT
    code = f"""
import torch, sys
sys.path.insert(0, {ROOT!r} + "/modern-srwm_b200")
from srwm_b200 import _lib as L
x, w, y = (torch.randn(*s, device="cuda") for s in ((1200, 132), (1032, 132), (260, 3200)))
v = torch.randn(132, 3200, device="cuda")
graph = torch.cuda.CUDAGraph()
torch.cuda.synchronize()
with torch.cuda.graph(graph):
    a, b = L.host().linear(x, w, None), L.host().linear(y, v, None)
for _ in range(2):
    x.normal_()
    graph.replay()
    for out, ref in ((a, x.double() @ w.double().t()), (b, y.double() @ v.double().t())):
        assert float((out.double() - ref).abs().max() / ref.abs().max()) < 3e-6
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
