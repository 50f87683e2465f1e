"""The debug build of the library (row checks that report through a status word instead of
faulting) on the GPU: the reporting path works, and the kernels raise no violation on sequence
lengths around their time-chunk length, on empty sequences and on strided views.

Runs in a child process because the build is chosen when the library is loaded
(``SRWM_B200_DEBUG=1``)."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r'''
import sys, torch
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[2])
import srwm_b200 as sb
from srwm_b200 import _lib as L
from srwm_b200 import layer_ops as lo
from conftest import srwm_inputs, delta_inputs
assert L.DEBUG_BUILD and L.LIB_PATH.endswith("libsrwm_b200_debug.so")
dev = torch.device("cuda", 0)
torch.cuda.set_device(dev)
ok, w = L.debug_status()
assert ok and w == 0, (ok, w)
# the reporting path: a check that must fail (no memory is touched by it)
L.check(L.load().srwm_b200_debug_selftest(None), "selftest")
ok, w = L.debug_status()
assert ok and (w >> 63) == 1 and ((w >> 48) & 0xff) == 255, hex(w)
assert L.debug_status() == (True, 0)            # cleared by the read
for E in (8, 16, 32, 64):
    for Ln in (0, 1, 15, 16, 17, 33):
        x, Ws, go = srwm_inputs(2, 3, Ln, E, 5)
        for dt in (torch.float32, torch.bfloat16):
            xd = x.permute(2, 0, 1, 3).contiguous().to(dev, dt).permute(1, 2, 0, 3)
            god = go.to(dev, dt)
            Wd = [t.to(dev) for t in Ws]
            out, saved = sb.srwm_forward(xd, *Wd)
            sb.srwm_backward(xd, saved, god, *Wd, restore_state=True)
            base = [t[:1].contiguous() for t in Wd]
            o2, sh, sv = lo.srwm_layer_forward(xd, base, None, None, True)
            if Ln > 0:
                lo.srwm_layer_backward(xd, sv, god, base, sh, None, True)
                lo.srwm_backward_detached(xd, sv, god, base[0], None, None, True)
        Q, K, V, B, W0, go = delta_inputs(2, 3, Ln, E, 6, "rand")
        for dt in (torch.float32, torch.bfloat16):
            Qd, Kd, Vd, Bd, god = (t.to(dev, dt) for t in (Q, K, V, B, go))
            W = W0.to(dev)
            out, saved = sb.delta_forward(Qd, Kd, Vd, Bd, W)
            sb.delta_backward(Qd, Kd, Vd, Bd, saved, god, W)
torch.cuda.synchronize()
ok, w = L.debug_status()
assert ok and w == 0, hex(w)
print("debug-build checks clean")
'''

GAVE_UP = r'''
import sys, torch
sys.path.insert(0, sys.argv[1])
from srwm_b200 import _lib as L
host = L.host()
assert L.DEBUG_BUILD
x, w = torch.randn(1200, 132, device="cuda"), torch.randn(1032, 132, device="cuda")
y, v = torch.randn(260, 3200, device="cuda"), torch.randn(132, 3200, device="cuda")        # a sum cut into parts
want = [(a.double() @ b.double().t()) for a, b in ((x, w), (y, v))]
tiles = 0
for (a, b), ref in zip(((x, w), (y, v)), want):
    for add in (None, torch.zeros(ref.shape, device="cuda")):
        assert L.load().srwm_b200_debug_gemm_tries(0) == 0
        out = host.linear(a, b, add)
        assert bool(out.isnan().all())
        assert L.load().srwm_b200_gemm_timeouts() > tiles
        tiles = L.load().srwm_b200_gemm_timeouts()
        assert L.load().srwm_b200_debug_gemm_tries(4000000) == 0
        try:
            host.linear(a, b, add)
            raise AssertionError("the call after one that gave up must fail")
        except L.SrwmError as e:
            assert e.code == L.ERR_TIMEOUT and "NaN" in str(e)
        assert float((host.linear(a, b, add).double() - ref).abs().max()) < 1e-3
        assert L.load().srwm_b200_gemm_timeouts() == tiles
print("gave up and said so")
'''

AGAIN = r'''
import sys, torch
sys.path.insert(0, sys.argv[1])
from srwm_b200 import _lib as L
M, N, K = 6652, 264, 8192            # 78 pairs of tiles: the first CTAs have another unit behind theirs
x, w = torch.randn(M, K, device="cuda"), torch.randn(N, K, device="cuda")
x[:256, K - 2] = float("inf")        # their whole tiles are summed again, to the end
assert L.DEBUG_BUILD and L.load().srwm_b200_debug_gemm_tries(30000) == 0
out = L.host().linear(x, w, None)
assert L.load().srwm_b200_gemm_timeouts() == 0
assert bool(out[:256].isinf().all()) and bool(out[256:].isfinite().all())
print("nobody gave up")
'''

CHUNKS = r'''
import sys, torch
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[2])
import srwm_b200 as sb
from srwm_b200 import _lib as L
from srwm_b200.layer_ops import delta_packed_backward, delta_packed_forward
from conftest import delta_inputs
for E, fwd, bwds in ((16, 2, (2, 3)), (32, 1, (1,)), (64, 1, (1,))):
    for Ln in (1, 15, 16, 17, 49):
        for dt in (torch.float32, torch.bfloat16):
            Q, K, V, B, go = (t.to("cuda", dt) for t in delta_inputs(2, 3, Ln, E, 6, "rand")[:4] + (torch.randn(2, 3, Ln, E),))
            for bad in (False, True):
                if bad:
                    V[1, 1, Ln // 2, 3] = float("inf")       # (the second, step-by-step run)
                W = torch.zeros(2, 3, E, E, device="cuda")
                out, saved = sb.delta_forward(Q, K, V, B, W, variant=fwd)
                for v in bwds:
                    sb.delta_backward(Q, K, V, B, saved, go, W.clone(), variant=v)
                W = torch.zeros(2, 3, E, E, device="cuda")
                rows = torch.cat([Q, K, V, B], -1)
                out, saved = delta_packed_forward(rows, W, 1e-5)
                delta_packed_backward(rows, saved, go, W, 1e-5)
assert L.debug_status() == (True, 0)
print("chunks clean")
'''


def test_chunk_kernels_stay_clean():
    """Plain and packed rows, every compiled configuration, finite and not."""
    assert "chunks clean" in _child(CHUNKS).stdout


def test_a_product_that_gives_up_says_so():
    """Every wait of the product's kernel runs out at once: NaN, and the next call fails."""
    r = _child(GAVE_UP)
    assert "gave up and said so" in r.stdout


def test_no_wait_runs_out_while_infinities_are_summed_again():
    """A product's waits with a limit of some 7 ms, a hundred times what they take, and infinities that take 70 ms."""
    assert "nobody gave up" in _child(AGAIN).stdout


def test_debug_build_reports_and_stays_clean():
    r = _child(CHILD)
    assert "debug-build checks clean" in r.stdout


def _child(code):
    lib = os.path.join(ROOT, "modern-srwm_b200", "srwm_b200", "libsrwm_b200_debug.so")
    if not os.path.exists(lib):
        sys.path.insert(0, os.path.join(ROOT, "modern-srwm_b200", "csrc"))
        import build as _build
        _build.build(debug=True)
    env = dict(os.environ, SRWM_B200_DEBUG="1")
    r = subprocess.run([sys.executable, "-c", code, os.path.join(ROOT, "modern-srwm_b200"), os.path.join(ROOT, "tests")],
                       capture_output=True, text=True, timeout=900, env=env)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return r
