"""GPU: the host-buffer path on states large enough for several chunks (8, 9 and 16 of them),
and just too small for any split, against the device-resident run, bit for bit: both run the
same kernels on the same tiles."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsteps", [1, 3])
@pytest.mark.parametrize("physics,N,n,dtype", [("wave", 5, 16, "f32"), ("maxwell", 5, 12, "f64"),
                                               ("wave", 9, 16, "f32"), ("wave", 6, 13, "f32")])
def test_chunked_host_path_equals_the_device_path(cuda, bb, physics, N, n, dtype, nsteps):
    import torch
    m = bb.uniform_tet_mesh(n)
    dt = torch.float32 if dtype == "f32" else torch.float64
    s = bb.DGSolver(m, N, physics, dtype=dt)
    q0 = torch.randn((s.nf, m.K, s.Np), dtype=dt, device=cuda,
                     generator=torch.Generator(cuda).manual_seed(N)) * 1e-2
    step = s.dt_cfl()
    qa, ra = q0.clone(), torch.zeros_like(q0)
    s.run(qa, ra, step, nsteps)
    hin = q0.cpu().pin_memory()
    hout = torch.full_like(hin, float("nan")).pin_memory()
    qd, rd = torch.empty_like(q0), torch.zeros_like(q0)
    for graph in (True, False):
        hout.fill_(float("nan"))
        s.run_host(hin, hout, qd, rd.zero_(), step, nsteps, graph=graph)
        torch.cuda.synchronize()
        assert torch.equal(hout, qa.cpu()) and torch.equal(qd, qa) and torch.equal(rd, ra)
    s.check()
