"""GPU: the specialised stage kernels' tables are made when a tile is chosen, also while a stream is
being captured (nothing of the choice itself is recorded), and serve a launch on another stream."""
import pytest

pytestmark = pytest.mark.gpu


def test_tile_chosen_during_a_capture(cuda, bb, monkeypatch):
    import torch
    from bbdg import context, solver as solver_module
    fresh = context.Context(0)  # no tables yet
    m = bb.uniform_tet_mesh(3)
    want = bb.DGSolver(m, 9, "wave", dtype=torch.float32)
    want.set_tile(2)
    q0 = torch.randn((4, m.K, want.Np), device=cuda, dtype=torch.float32,
                     generator=torch.Generator(cuda).manual_seed(4)) * 1e-2
    qa, ra = q0.clone(), torch.zeros_like(q0)
    want.run(qa, ra, want.dt_cfl(), 2)
    with monkeypatch.context() as mp:
        mp.setattr(solver_module, "get_context", lambda device=None: fresh)
        s = bb.DGSolver(m, 9, "wave", dtype=torch.float32)
    assert s.ctx is fresh
    x = torch.zeros(4, device=cuda)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x += 1
        s.set_tile(2)
    assert s.kernel == "specialised" and s.tile[0] == 2
    g.replay()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    qb, rb = q0.clone(), torch.zeros_like(q0)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        s.run(qb, rb, s.dt_cfl(), 2)
    torch.cuda.synchronize()
    assert torch.equal(qa, qb) and torch.equal(ra, rb) and torch.equal(x, torch.ones_like(x))
    s.check()
    s.close()
    fresh.close()
