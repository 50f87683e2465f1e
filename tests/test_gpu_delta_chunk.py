"""The chunked delta-rule kernels (16 steps at a time on the tensor cores) against the float64 oracle
where they can go wrong: lengths around one and two chunks and around the ring of prepared chunks, a
carried state, both element types, dense and time-major rows."""
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
