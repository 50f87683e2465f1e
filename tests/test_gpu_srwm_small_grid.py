"""The SRWM forward that gives w_b a warp of its own (the choice for small grids) against the kernel of the same head
size that larger grids use: outputs, saved tensors and final state at lengths around one and two chunks, plain and in
the layer-level form with resets.  At d_head 64 both add in the same order, so the results are the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
IDS = {16: (2, 1), 32: (3, 1), 64: (2, 1)}      # head size -> (small-grid id, the other)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mode", ["plain", "layer", "resets"])
@pytest.mark.parametrize("E", [16, 32, 64])
@pytest.mark.parametrize("L", [1, 15, 16, 17, 33])
def test_small_grid_forward(E, L, mode, dtype):
    import srwm_b200 as sb
    from srwm_b200 import layer_ops as lo
    d = torch.device("cuda", 0)
    N, H = 3, 2
    g = torch.Generator(device=d).manual_seed(L + E)
    x = torch.randn(N, H, L, E, device=d, generator=g).to(dtype)
    base = [torch.randn(1, H, E, w, device=d, generator=g) * E ** -0.5 for w in (E, E, E, 4)]
    shift = [torch.randn(N, H, E, w, device=d, generator=g) * 0.1 * E ** -0.5 for w in (E, E, E, 4)]
    done = torch.rand(N, L, device=d, generator=g) < 0.2 if mode == "resets" else None
    res = []
    for v in IDS[E]:
        if mode == "plain":
            W = [b.repeat(N, 1, 1, 1) for b in base]
            out, saved = sb.srwm_forward(x, *W, variant=v)
            res.append([out, *saved, *W])
        else:
            out, state, saved = lo.srwm_layer_forward(x, base, shift, done, True, variant=v)
            res.append([out, *saved, *state])
    for a, b in zip(*res):
        if E == 64:
            assert torch.equal(a, b)
        else:
            tol = 8e-3 if a.dtype == torch.bfloat16 else 5e-4 if mode == "resets" else 2e-5
            assert float((a.float() - b.float()).abs().max()) <= tol * float(b.float().abs().max())
