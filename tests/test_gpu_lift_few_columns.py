"""GPU: the table-driven lift kernels give every column the same bits whatever the number of
columns: their tiles hold fewer elements when there are too few columns for the whole GPU."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,dtype", [(1, "f64"), (7, "f64"), (9, "f64"), (10, "f64"), (20, "f64"),
                                     (13, "f32"), (17, "f32")])
def test_columns_do_not_depend_on_their_number(cuda, bb, N, dtype):
    import torch
    dt = torch.float32 if dtype == "f32" else torch.float64
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    most = 16 * sms + 5
    gen = torch.Generator(cuda).manual_seed(N)
    faces = torch.rand((most, 4 * bb.np2(N)), dtype=dt, device=cuda, generator=gen) - 0.5
    one = faces[:, :bb.np2(N)].contiguous()
    L = bb.BernsteinLift(N)

    def lifts(K):
        a = torch.full((K, bb.np3(N)), float("nan"), dtype=dt, device=cuda)
        b = a.clone()
        bb.mul_(a, L, faces[:K].contiguous())
        bb.operators.face_lift_multiply_(b, L, one[:K].contiguous())
        return a, b

    want = lifts(most)
    # a single lifted face is the full lift of columns that are zero on the other three
    padded = torch.zeros_like(faces)
    padded[:, 3 * bb.np2(N):] = one
    full = bb.mul_(torch.empty_like(want[0]), L, padded)
    tol = 1e-12 if dtype == "f64" else 1e-4
    assert (full - want[1]).abs().max() <= tol * want[1].abs().max()
    for K in (1, 2, 15, 16, 17, sms - 1, sms, sms + 1, 2 * sms + 1, 4 * sms - 1, 8 * sms + 3,
              16 * sms - 1, 16 * sms):
        for got, w in zip(lifts(K), want):
            assert torch.equal(got, w[:K]), K
