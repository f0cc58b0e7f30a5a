"""GPU: the split-K GEMM adds its partial tiles with vector reductions where the output rows are
16-byte aligned, else float by float: ragged sizes, row lengths and a misaligned output, on small
whole-number operands (every partial sum is an integer below 2^24: exact in any order)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(128, 256, 512), (1, 1, 192), (130, 4, 256), (33, 37, 320),
                                   (200, 260, 1024), (127, 129, 648), (513, 336, 256)])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_exact_sums(cuda, M, N, K, offset):
    import torch
    from bbdg import mlp
    g = torch.Generator(device="cuda").manual_seed(M + N)
    A = torch.randint(-8, 9, (M, K), generator=g, device=cuda).bfloat16()
    B = torch.randint(-8, 9, (N, K), generator=g, device=cuda).bfloat16()
    buf = torch.full((M * N + 8,), 3.0, device=cuda)
    C = buf[4 + offset:4 + offset + M * N].view(M, N)
    for kt_per in (1, 2, 3):
        buf.fill_(3.0)
        mlp.gemm_bf16(A, B, out_f32=C, kt_per=kt_per)
        # one part holds all of K: nothing is split, and the output is stored, not added to
        want = (3.0 if kt_per < (K + 63) // 64 else 0.0) + A.double() @ B.double().T
        assert torch.equal(C.double(), want)
        # nothing beside the output was touched
        assert (buf[:4 + offset] == 3.0).all() and (buf[4 + offset + M * N:] == 3.0).all()
    assert mlp.device_status() == 0
