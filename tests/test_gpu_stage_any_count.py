"""Degree-specialised stage kernels on element counts that are no multiple of their tile.

The last tile of a mesh is then partial, and where the field rows do not start on 16-byte
boundaries (an odd number of coefficients) tiles are copied 8 or 4 bytes at a time. The meshes
are a periodic cube plus 0 to 3 lone elements whose faces meet each other, so that every
remainder of K modulo 4 occurs; the reference is the generic kernel in FP64.
"""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mesh_with_lone_elements(bb, n, extra):
    """uniform_tet_mesh(n) and `extra` copies of its first element, face 0 of each meeting its
    face 1 and face 2 its face 3 (orientation (0, 1, 2), an involution)."""
    m = bb.uniform_tet_mesh(n)
    K = m.K
    nbr = np.concatenate([m.nbr, np.repeat(np.arange(K, K + extra)[:, None], 4, axis=1)])
    nbf = np.concatenate([m.nbr_face, np.tile([[1, 0, 3, 2]], (extra, 1))])
    ori = np.concatenate([m.orient, np.zeros((extra, 4), m.orient.dtype)])
    geo = np.concatenate([m.geo, np.repeat(m.geo[:1], extra, axis=0)])
    return dataclasses.replace(m, K=K + extra, nbr=nbr, nbr_face=nbf, orient=ori, geo=geo,
                               conn=bb.mesh.pack_connectivity(nbr, nbf, ori))


def rel(a, b):
    return [float((x.double() - y).norm() / y.norm()) for x, y in zip(a, b)]


# degrees with Np a multiple of 4 (bulk copies always), Np = 2 mod 4 and Np odd
@pytest.mark.parametrize("physics,N", [("wave", 3), ("maxwell", 3), ("wave", 12), ("maxwell", 12),
                                       ("wave", 13), ("maxwell", 13), ("wave", 14),
                                       ("maxwell", 14), ("wave", 15), ("maxwell", 15), ("wave", 4), ("maxwell", 4), ("wave", 5), ("maxwell", 6),
                                       ("wave", 8), ("maxwell", 8), ("wave", 9), ("maxwell", 10),
                                       ("wave", 11)])
@pytest.mark.parametrize("n,extra", [(2, 0), (2, 1), (2, 2), (2, 3), (7, 1)])
def test_any_element_count(cuda, bb, physics, N, n, extra):
    """The right-hand side of a random state and two LSRK steps against FP64: 1e-5 per field,
    the repository's FP32 tolerance. K = 48 .. 51 is one or a few tiles, K = 2,059 (7^3 x 6 + 1)
    several per block with a partial last one."""
    import torch
    m = mesh_with_lone_elements(bb, n, extra)
    s = bb.DGSolver(m, N, physics, dtype=torch.float32, tau=1.0)
    assert s.kernel == "specialised"
    d = bb.DGSolver(m, N, physics, dtype=torch.float64, tau=1.0)
    gen = torch.Generator(device=cuda).manual_seed(10 * N + extra)
    q = torch.rand((s.nf, m.K, s.Np), generator=gen, device=cuda) * 2 - 1
    q64 = q.double()
    err = rel(s.rhs(q), d.rhs(q64))
    assert max(err) < 1e-5, err
    dt = s.dt_cfl()
    s.run(q, torch.zeros_like(q), dt, 2)
    s.check()
    d.run(q64, torch.zeros_like(q64), dt, 2)
    err = rel(q, q64)
    assert max(err) < 1e-5, err


@pytest.mark.parametrize("physics", ["wave", "maxwell"])
@pytest.mark.parametrize("N", [12, 13, 14, 15])
def test_high_degrees_equal_the_generic_kernel(cuda, bb, physics, N):
    """From degree 12 on the specialised kernel does the generic kernel's arithmetic: the same
    bits, in both penalty modes and with a partial last tile."""
    import torch
    m = mesh_with_lone_elements(bb, 3, 1)
    for tau in (1.0, 0.0):
        s = bb.DGSolver(m, N, physics, dtype=torch.float32, tau=tau)
        assert s.kernel == "specialised"
        gen = torch.Generator(device=cuda).manual_seed(N)
        q0 = torch.rand((s.nf, m.K, s.Np), generator=gen, device=cuda) * 2 - 1
        out = []
        for kind in ("specialised", "generic"):
            s.set_kernel(kind)
            q = q0.clone()
            rhs = s.rhs(q)
            s.run(q, torch.zeros_like(q), 1e-3 * s.dt_cfl(), 2)
            s.check()
            out.append((rhs, q))
        assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


@pytest.mark.parametrize("physics,N,dtype", [("wave", 9, "float32"), ("maxwell", 5, "float32"),
                                             ("wave", 13, "float32"), ("advection", 4, "float32"),
                                             ("maxwell", 3, "float64"), ("wave", 20, "float64")])
def test_a_step_ignores_the_register_it_starts_with(cuda, bb, physics, N, dtype):
    """The LSRK register is scratch within a step: NaN in it before the step changes nothing."""
    import torch
    m = bb.uniform_tet_mesh(3)
    s = bb.DGSolver(m, N, physics, dtype=getattr(torch, dtype), tau=1.0)
    gen = torch.Generator(device=cuda).manual_seed(N)
    q0 = torch.rand((s.nf, m.K, s.Np), generator=gen, device=cuda, dtype=s.dtype)
    out = []
    for fill in (0.0, float("nan")):
        q, r = q0.clone(), torch.full_like(q0, fill)
        s.run(q, r, 0.1 * s.dt_cfl(), 2)
        s.check()
        out.append((q, r))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
