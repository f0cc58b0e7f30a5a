"""GPU: the closure's features and update give an element the same values whatever the number of
elements: a block takes one to eight of them, by how many there are for the whole GPU."""
import pytest

pytestmark = pytest.mark.gpu


def counts(sms):
    return (1, 2, 4 * sms - 1, 4 * sms, 8 * sms - 1, 8 * sms + 3, 16 * sms - 1, 16 * sms + 1,
            32 * sms - 1, 32 * sms + 5)


@pytest.mark.parametrize("N,nf,dtype", [(1, 4, "f64"), (2, 6, "f32"), (5, 6, "f64"), (7, 4, "f32")])
def test_features(cuda, bb, N, nf, dtype):
    import torch
    from bbdg import mlp
    ks = counts(torch.cuda.get_device_properties(0).multi_processor_count)
    dt = torch.float32 if dtype == "f32" else torch.float64
    gen = torch.Generator(cuda).manual_seed(N)
    q = torch.randn((nf, ks[-1], bb.np3(N)), device=cuda, dtype=dt, generator=gen)
    # every face meets the element itself, on some face and in some orientation
    e = torch.arange(ks[-1], device=cuda).view(-1, 1)
    face = torch.randint(0, 4, (ks[-1], 4), device=cuda, generator=gen)
    orient = torch.randint(0, 6, (ks[-1], 4), device=cuda, generator=gen)
    conn = ((e << 5) | (face << 3) | orient).to(torch.int32)
    want = None
    for K in ks:
        X, _ = mlp.closure_features(N, nf, conn[:K].reshape(-1).contiguous(),
                                    q[:, :K].contiguous(), 0.5)
        if want is not None:
            assert torch.equal(X[:want.shape[0]], want), K
        want = X
    h = (q.float() * 0.5).bfloat16()
    assert torch.equal(want[:, :nf * bb.np3(N)], h.permute(1, 0, 2).reshape(ks[-1], -1))


@pytest.mark.parametrize("N,nf,dtype", [(1, 1, "f64"), (3, 2, "f64"), (5, 6, "f32"), (7, 4, "f64")])
def test_apply(cuda, bb, N, nf, dtype):
    import torch
    from bbdg import mlp
    ks = counts(torch.cuda.get_device_properties(0).multi_processor_count)
    dt = torch.float32 if dtype == "f32" else torch.float64
    gen = torch.Generator(cuda).manual_seed(N)
    q0 = torch.randn((nf, ks[-1], bb.np3(N)), device=cuda, dtype=dt, generator=gen)
    Y = torch.randn((ks[-1], nf * bb.np3(N)), device=cuda, generator=gen)
    want = None
    for K in ks:
        q = q0[:, :K].clone(memory_format=torch.contiguous_format)
        mlp.closure_apply(N, nf, 0.25, Y[:K].contiguous(), q)
        if want is not None:
            assert torch.equal(q[:, :want.shape[1]], want), K
        want = q
    # a product by a power of two is exact: one rounding to FP32, one to the state's type
    sum32 = q0.float() + 0.25 * Y.view(ks[-1], nf, -1).permute(1, 0, 2)
    assert torch.equal(want, sum32.to(dt))
