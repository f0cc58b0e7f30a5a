"""GPU: the combined operator call with outputs in the memory of its inputs, in double. At N = 9 a
face column (4 Nfp) and a volume column (Np) have the same length, so a gradient can be stored where
the face columns are."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 384, 5001])
@pytest.mark.parametrize("into", ["dr", "ds", "dt", "lift", "all"])
def test_outputs_over_inputs(cuda, bb, K, into):
    import torch
    N = 9
    assert bb.np3(N) == 4 * bb.np2(N)
    gen = torch.Generator(cuda).manual_seed(K)
    x0, f0 = (torch.rand((K, bb.np3(N)), dtype=torch.float64, device=cuda, generator=gen)
              for _ in range(2))
    want = [torch.empty_like(x0) for _ in range(4)]
    bb.fused_apply_(*want, N, x0, f0)
    # a gradient over the face columns, or the lift over the volume columns; "all": a gradient over
    # the volume columns it comes from and the lift over its own face columns
    names = ["dr", "ds", "dt", "lift"]
    for place in [0, 1, 2] if into == "all" else [names.index(into)]:
        x, f = x0.clone(), f0.clone()
        out = [torch.empty_like(x0) for _ in range(4)]
        if into == "all":
            out[place], out[3] = x, f
        else:
            out[place] = x if into == "lift" else f
        bb.fused_apply_(*out, N, x, f)
        for got, w in zip(out, want):
            assert torch.equal(got, w)
