"""GPU: the closure's feature gather and update where the element count is no multiple of the
elements a block takes, in both precisions and at the lowest and highest degree.

Both are one multiplication (or one multiply-add) and a rounding per value. The features are
compared exactly; the update may differ from the separate product and sum by one rounding of
the product, at most 2^-24 of it, plus one rounding of the sum in the state's precision.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _face_tables(bb, N):
    """Volume index of face f's node m (face-local (a, b), b outer)."""
    from oracle import dense
    idx = {t[:3]: n for n, t in enumerate(dense.lut3(N))}
    faces = np.zeros((4, bb.np2(N)), np.int64)
    for f in range(4):
        m = 0
        for b in range(N + 1):
            for a in range(N + 1 - b):
                faces[f, m] = idx[((a, 0, b), (N - a - b, a, b), (0, a, b), (a, b, 0))[f]]
                m += 1
    return faces


@pytest.mark.parametrize("N,nf,dtype", [(1, 4, "f32"), (5, 6, "f32"), (5, 6, "f64"),
                                        (20, 4, "f32")])
def test_features_element_remainders(cuda, bb, N, nf, dtype):
    import torch
    from bbdg import mlp
    mesh = bb.uniform_tet_mesh(3)                       # 162 elements: remainder 2 of 8
    K, Np, Nfp = mesh.K, bb.np3(N), bb.np2(N)
    assert K % 8 != 0
    dt = torch.float32 if dtype == "f32" else torch.float64
    q = torch.randn((nf, K, Np), device=cuda, dtype=dt, generator=torch.Generator(cuda).manual_seed(N))
    conn = torch.tensor(mesh.conn.reshape(-1), dtype=torch.int32, device=cuda)
    X = mlp.closure_features(N, nf, conn, q, 0.5)
    X = X[0] if isinstance(X, tuple) else X
    torch.cuda.synchronize()
    h = (q.cpu().float() * 0.5).bfloat16()
    got = X.cpu()
    assert torch.equal(got[:, :nf * Np], h.permute(1, 0, 2).reshape(K, nf * Np))
    faces = _face_tables(bb, N)
    c = np.asarray(mesh.conn, np.int64).reshape(K, 4)
    ext = got[:, nf * Np:].reshape(K, 4, nf, Nfp)
    for f in range(4):
        for e in range(K):
            nbr, nface = int(c[e, f] >> 5), int(c[e, f] >> 3) & 3
            # the neighbour's face values, each exactly once (the pairing is a permutation)
            want = h[:, nbr, faces[nface]]
            assert torch.equal(ext[e, f].float().sort(dim=1)[0], want.float().sort(dim=1)[0])


@pytest.mark.parametrize("K", [1, 3, 5, 102])
@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_apply_element_remainders(cuda, bb, K, dtype):
    import torch
    from bbdg import mlp
    N, nf = 4, 4
    Np = bb.np3(N)
    dt = torch.float32 if dtype == "f32" else torch.float64
    q = torch.randn((nf, K, Np), device=cuda, dtype=dt)
    Y = torch.randn((K, nf * Np), device=cuda)
    q0, d = q.cpu().float().double(), Y.cpu().double().reshape(K, nf, Np).permute(1, 0, 2) * 0.25
    mlp.closure_apply(N, nf, 0.25, Y, q)
    torch.cuda.synchronize()
    # the sum is taken in single precision for both state types
    err = (q.cpu().double() - (q0 + d)).abs()
    assert bool((err <= 2.0 ** -24 * (d.abs() + (q0 + d).abs() * 1.01)).all())
