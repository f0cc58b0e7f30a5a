"""GPU: the combined operator call gives the bits of the gradient and lift calls whatever the number
of columns: one launch serves both operators where few columns leave room for that."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,dtype", [(1, "f64"), (3, "f64"), (7, "f64"), (9, "f64"), (16, "f64"),
                                     (17, "f64"), (20, "f64"), (16, "f32"), (20, "f32"), (5, "f32")])
def test_equals_the_separate_calls(cuda, bb, N, dtype):
    import torch
    dt = torch.float32 if dtype == "f32" else torch.float64
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ks = (1, 2, 17, sms - 1, 2 * sms, 2 * sms + 1, 4 * sms + 1, 8 * sms - 1, 32 * sms + 3)
    gen = torch.Generator(cuda).manual_seed(N)
    x = torch.rand((max(ks), bb.np3(N)), dtype=dt, device=cuda, generator=gen) - 0.5
    faces = torch.rand((max(ks), 4 * bb.np2(N)), dtype=dt, device=cuda, generator=gen) - 0.5
    L = bb.BernsteinLift(N)
    want = [torch.empty_like(x) for _ in range(4)]
    bb.grad_(*want[:3], N, x)
    bb.mul_(want[3], L, faces)
    for K in ks:
        out = [torch.full_like(x[:K], float("nan")) for _ in range(4)]
        bb.fused_apply_(*out, N, x[:K].contiguous(), faces[:K].contiguous())
        for got, w in zip(out, want):
            assert torch.equal(got, w[:K]), K
