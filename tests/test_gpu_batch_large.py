"""GPU: batches whose problems take every route of a step at once. Small problems run on the side
streams, the generic ones beside them on the caller's stream, and those that fill the GPU by
themselves one after the other behind the join; each ends bitwise equal to a single solver running
the same kernel."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
def test_small_generic_and_large_problems_together(cuda, bb, graph):
    import torch
    from bbdg.batch import BatchSolver, ProblemSpec
    # large: two tiles per resident block and more (8 elements a tile at wave N = 5, 2 at Maxwell
    # N = 9, at most four blocks on each of the SMs); small and generic ones between them
    specs = [ProblemSpec("wave", 5, 13, seed=1), ProblemSpec("wave", 5, 3, seed=2),
             ProblemSpec("advection", 6, 4, seed=3), ProblemSpec("maxwell", 9, 8, seed=4),
             ProblemSpec("maxwell", 4, 3, seed=5), ProblemSpec("wave", 2, 4, seed=6)]
    gen = torch.Generator().manual_seed(9)
    nf = {"wave": 4, "maxwell": 6, "advection": 1}
    states = [torch.randn((nf[s.physics], 6 * s.n ** 3, bb.np3(s.N)), generator=gen).numpy() * 1e-2
              for s in specs]
    B = BatchSolver(specs, dtype=torch.float32, states=states)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert B.meshes[0].K >= 2 * 8 * 4 * sms and B.meshes[3].K >= 2 * 2 * 4 * sms
    q0 = [q.clone() for q in B.q]
    for n in (1, 2):  # the second call starts from traces extracted anew
        B.run(n, graph=graph)
    torch.cuda.synchronize()
    for p, spec in enumerate(specs):
        s = bb.DGSolver(B.meshes[p], spec.N, spec.physics, dtype=torch.float32, tau=spec.tau)
        if s.kernel == "generic":
            s.set_tile(B.tile(spec.physics, spec.N), 256)
        q, r = q0[p].clone(), torch.zeros_like(q0[p])
        s.run(q, r, B.dt(p), 3, graph=False)
        torch.cuda.synchronize()
        assert torch.equal(q, B.q[p]) and torch.equal(r, B.res[p]), (p, s.kernel)
