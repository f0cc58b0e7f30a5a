"""GPU: the host-buffer path with the most chunks it takes (24, from 190 MB of state on) and with
ten and thirteen, against the device-resident run, bit for bit. The chunk count is read from the launches of a
replayed step: one trace extraction and five stages per chunk."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("physics,N,n,dtype,chunks", [("wave", 9, 21, "f32", 24),
                                                      ("wave", 9, 12, "f32", 10),
                                                      ("wave", 3, 25, "f64", 13)])
def test_chunked_steps_equal_the_device_path(cuda, bb, physics, N, n, dtype, chunks):
    import torch
    m = bb.uniform_tet_mesh(n)
    dt = torch.float32 if dtype == "f32" else torch.float64
    s = bb.DGSolver(m, N, physics, dtype=dt)
    q0 = torch.randn((s.nf, m.K, s.Np), dtype=dt, device=cuda,
                     generator=torch.Generator(cuda).manual_seed(n)) * 1e-2
    step = s.dt_cfl()
    hin = q0.cpu().pin_memory()
    hout = torch.empty_like(hin).pin_memory()
    qd, rd = torch.empty_like(q0), torch.zeros_like(q0)
    s.run_host(hin, hout, qd, rd, step, 1)
    torch.cuda.synchronize()
    before = s.ctx.launch_count()
    s.run_host(hin, hout, qd, rd.zero_(), step, 1)
    assert s.ctx.launch_count() - before == 6 * chunks
    for nsteps in (1, 3):
        qa, ra = q0.clone(), torch.zeros_like(q0)
        s.run(qa, ra, step, nsteps)
        want = qa.cpu()
        for graph in (True, False):
            hout.fill_(float("nan"))
            s.run_host(hin, hout, qd, rd.zero_(), step, nsteps, graph=graph)
            torch.cuda.synchronize()
            assert torch.equal(hout, want) and torch.equal(qd, qa) and torch.equal(rd, ra)
    s.check()
