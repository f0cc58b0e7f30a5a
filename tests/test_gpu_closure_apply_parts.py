"""GPU: the closure's update with an element's values shared out over several blocks, at the numbers of
elements around which it no longer is (four elements a block, 16 blocks for every SM)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm", [32, 64])
@pytest.mark.parametrize("more", [-5, 0, 3])
@pytest.mark.parametrize("N,nf,dtype", [(5, 6, "f32"), (5, 6, "f64"), (6, 4, "f64")])
def test_apply(cuda, bb, N, nf, dtype, per_sm, more):
    import torch
    from bbdg import mlp
    K = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    dt = torch.float32 if dtype == "f32" else torch.float64
    gen = torch.Generator(cuda).manual_seed(K)
    q = torch.randn((nf, K, bb.np3(N)), device=cuda, dtype=dt, generator=gen)
    Y = torch.randn((K, nf * bb.np3(N)), device=cuda, generator=gen)
    # a product by a power of two is exact: one rounding to FP32, one to the state's type
    want = (q.float() + 0.25 * Y.view(K, nf, -1).permute(1, 0, 2)).to(dt)
    mlp.closure_apply(N, nf, 0.25, Y, q)
    assert torch.equal(q, want)
