"""GPU: solvers that have a specialised kernel but run the generic one, because it was asked for or
because a buffer is not on a 16-byte boundary, run it on the generic kernel's own tile."""
import pytest

pytestmark = pytest.mark.gpu


def offset_copy(x, by):
    import torch
    buf = torch.empty(x.numel() + 4, dtype=x.dtype, device=x.device)
    out = buf[by:by + x.numel()].view(x.shape)
    out.copy_(x)
    return out


@pytest.mark.parametrize("physics,N,tiles", [("wave", 9, (4, 2)), ("maxwell", 5, (4, 8))])
def test_generic_tile_does_not_depend_on_the_specialised_one(cuda, bb, physics, N, tiles):
    import torch
    m = bb.uniform_tet_mesh(6)
    got = set()
    for e in tiles:
        s = bb.DGSolver(m, N, physics, dtype=torch.float32)
        s.set_tile(e)
        assert s.kernel == "specialised" and s.tile[0] == e
        s.set_kernel("generic")
        assert s.kernel == "generic"
        got.add(s.tile)
    assert len(got) == 1


@pytest.mark.parametrize("physics,N,n", [("wave", 3, 5), ("maxwell", 3, 5), ("wave", 9, 5),
                                         ("maxwell", 10, 3), ("wave", 12, 3), ("maxwell", 13, 2)])
@pytest.mark.parametrize("by", [1, 2])
def test_misaligned_buffers(cuda, bb, physics, N, n, by):
    import torch
    m = bb.uniform_tet_mesh(n)
    s = bb.DGSolver(m, N, physics, dtype=torch.float32)
    assert s.kernel == "specialised"
    tile = s.tile
    g = bb.DGSolver(m, N, physics, dtype=torch.float32)
    g.set_kernel("generic")
    q0 = torch.randn((s.nf, m.K, s.Np), device=cuda,
                     generator=torch.Generator(cuda).manual_seed(N)) * 1e-2
    step = s.dt_cfl()
    want, r = q0.clone(), torch.zeros_like(q0)
    g.run(want, r, step, 2)
    rhs = g.rhs(q0)
    fast, rf = q0.clone(), torch.zeros_like(q0)
    s.run(fast, rf, step, 2)
    for graph in (True, False):
        q, res = offset_copy(q0, by), offset_copy(torch.zeros_like(q0), by)
        s.run(q, res, step, 2, graph=graph)
        assert torch.equal(q, want) and torch.equal(res, r)
    q, res = q0.clone(), offset_copy(torch.zeros_like(q0), by)  # one of the two is enough
    s.run(q, res, step, 2)
    assert torch.equal(q, want)
    assert torch.equal(s.rhs(offset_copy(q0, by)), rhs)
    assert torch.equal(s.rhs(q0, out=offset_copy(q0, by)), rhs)
    hin = q0.cpu().pin_memory()
    hout = torch.empty_like(hin).pin_memory()
    s.run_host(hin, hout, offset_copy(q0, by), offset_copy(torch.zeros_like(q0), by), step, 2)
    torch.cuda.synchronize()
    assert torch.equal(hout, want.cpu())
    # the solver itself is as it was
    assert s.kernel == "specialised" and s.tile == tile
    q, res = q0.clone(), torch.zeros_like(q0)
    s.run(q, res, step, 2)
    assert torch.equal(q, fast)
    s.check()
