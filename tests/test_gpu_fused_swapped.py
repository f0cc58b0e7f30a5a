"""GPU: the combined operator call with its inputs' memory exchanged for its outputs': at N = 9 a face
column and a volume column have the same length, so a gradient can be stored where the face columns
are and the lift where the volume columns are."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("K", [1, 384, 5001])
@pytest.mark.parametrize("place", [0, 1, 2])
def test_gradient_and_lift_over_each_others_input(cuda, bb, K, place, dtype):
    import torch
    N = 9
    gen = torch.Generator(cuda).manual_seed(K)
    x0, f0 = (torch.rand((K, bb.np3(N)), dtype=getattr(torch, dtype), device=cuda, generator=gen)
              for _ in range(2))
    want = [torch.empty_like(x0) for _ in range(4)]
    bb.fused_apply_(*want, N, x0, f0)
    x, f = x0.clone(), f0.clone()
    out = [torch.empty_like(x0) for _ in range(4)]
    out[place], out[3] = f, x
    bb.fused_apply_(*out, N, x, f)
    for got, w in zip(out, want):
        assert torch.equal(got, w)
