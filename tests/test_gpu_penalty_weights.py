"""GPU: the face penalty weights tau |n| and tau / |n| of the specialised FP32 stage kernels, rounded
as the generic kernel's (a square root and a division to the nearest).

One element holds 1 in one field and every other coefficient of the mesh is zero, so a neighbour that
meets it on one face has no volume term, and lift inputs that are constant on that face and zero on
the others. With normals (0, a, b) of integer length c = |n| times a power of two, tau a power of two
(or one times c, all faces with the same c, which makes tau / |n| a power of two) and 1/J = 1, every
operation up to layer 0 of that face's stack is exact in FP32 (integers below 2^24 times a power of
two), and the right-hand side there is an exact number, if the weights are."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TRIPLES = [(3, 4, 5), (5, 12, 13), (8, 15, 17), (7, 24, 25), (20, 21, 29), (12, 35, 37), (9, 40, 41),
           (28, 45, 53), (11, 60, 61), (33, 56, 65), (16, 63, 65), (48, 55, 73), (13, 84, 85),
           (36, 77, 85), (39, 80, 89), (65, 72, 97), (20, 99, 101), (60, 91, 109), (15, 112, 113),
           (44, 117, 125), (88, 105, 137), (24, 143, 145), (51, 140, 149), (85, 132, 157)]


def geometry(m, s, rng, triples):
    """Overwrites the solver's geometry; returns the (K, 4, 3) triples a, b, c of the faces."""
    import torch
    pick = rng.integers(0, len(triples), (m.K, 4))
    t = np.array(triples)[pick] * (2.0 ** rng.integers(-6, 3, (m.K, 4)))[..., None]
    geo = np.zeros((m.K, 24))
    geo[:, :9] = rng.standard_normal((m.K, 9))
    geo[:, 9] = geo[:, 10] = 1.0
    geo[:, 16:20], geo[:, 20:24] = t[..., 0], t[..., 1]
    s.geo.copy_(torch.as_tensor(geo.reshape(-1), dtype=torch.float32))
    return t


def check(m, s, N, field, flux):
    """flux(e, f): the exact lift input of field `field` on face f of element e, whose neighbour
    there holds 1 in that field."""
    # coefficients of layer 0 of each face, by face node, and the constant's image under L0
    at = {a: p for p, a in enumerate((i, j, k) for k in range(N + 1) for j in range(N + 1 - k)
                                     for i in range(N + 1 - j - k))}
    nodes = [(a, b) for b in range(N + 1) for a in range(N + 1 - b)]
    vol = [lambda a, b: (a, 0, b), lambda a, b: (N - a - b, a, b), lambda a, b: (0, a, b),
           lambda a, b: (a, b, 0)]

    def image(i, j):
        k = N - i - j
        return 0.5 * ((i + 1) ** 2 + (j + 1) ** 2 + (k + 1) ** 2 + (i + 1) * (j + k)
                      + (j + 1) * (i + k) + (k + 1) * (i + j))

    checked = 0
    for src in range(0, m.K, 7):
        q = s.zeros()
        q[field, src] = 1.0
        rhs = s.rhs(q)[field].double().cpu().numpy()
        for e in set(m.nbr[src]):
            faces = [f for f in range(4) if m.nbr[e, f] == src]
            if e == src or len(faces) != 1:
                continue
            p = [at[vol[faces[0]](a, b)] for a, b in nodes]
            want = np.array([image(a, b) for a, b in nodes]) * flux(e, faces[0])
            assert np.array_equal(rhs[e, p], want), (src, e, faces[0])
            checked += 1
    assert checked >= 100


@pytest.mark.parametrize("physics", ["wave", "maxwell"])
@pytest.mark.parametrize("N", range(3, 16))
def test_exact_lengths_give_exact_products(cuda, bb, physics, N):
    import torch
    m = bb.uniform_tet_mesh(4)
    s = bb.DGSolver(m, N, physics, dtype=torch.float32, tau=0.5)
    assert s.kernel == "specialised"
    t = geometry(m, s, np.random.default_rng(N), TRIPLES)
    # field 0 is p, or H_x with n_x = 0: its flux is tau |n| / 2
    check(m, s, N, 0, lambda e, f: 0.25 * t[e, f, 2])


@pytest.mark.parametrize("physics", ["wave", "maxwell"])
@pytest.mark.parametrize("N", range(3, 16))
@pytest.mark.parametrize("triple", [TRIPLES[1], TRIPLES[8], TRIPLES[12], TRIPLES[23]])
def test_exact_lengths_give_exact_quotients(cuda, bb, physics, N, triple):
    import torch
    m = bb.uniform_tet_mesh(4)
    c = triple[2]
    s = bb.DGSolver(m, N, physics, dtype=torch.float32, tau=c)
    assert s.kernel == "specialised"
    t = geometry(m, s, np.random.default_rng(N + c), [triple])
    if physics == "wave":  # v: n_y times the scalar flux tau / |n| n_y / 2
        check(m, s, N, 2, lambda e, f: 0.5 * c / t[e, f, 2] * t[e, f, 0] ** 2)
    else:  # H_y: tau |n| / 2 - tau / |n| n_y^2 / 2
        check(m, s, N, 1, lambda e, f: 0.5 * c * t[e, f, 2] - 0.5 * c / t[e, f, 2] * t[e, f, 0] ** 2)
