"""GPU: batches in double whose generic problems need both launches of a stage (tiles that fill an
SM's shared memory, and smaller ones), against single solvers on the same tiles, bit for bit."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("kinds", [
    # both launches, the large tiles first, last and between
    [("maxwell", 12, 2, None), ("wave", 5, 4, None), ("maxwell", 11, 2, None), ("wave", 3, 3, None)],
    # only large ones; only small ones
    [("maxwell", 13, 2, None), ("wave", 15, 2, None)],
    [("wave", 4, 2, None), ("maxwell", 3, 2, None)],
    # a tile chosen by hand that fills an SM beside default ones
    [("wave", 7, 3, 4), ("advection", 6, 2, None), ("wave", 2, 3, None)]])
def test_lanes_equal_single_solvers(cuda, bb, kinds, graph):
    import torch
    from bbdg.batch import BatchSolver, ProblemSpec
    nf = {"wave": 4, "maxwell": 6, "advection": 1}
    specs = [ProblemSpec(p, N, n, seed=i) for i, (p, N, n, _) in enumerate(kinds)]
    gen = torch.Generator().manual_seed(3)
    states = [torch.randn((nf[s.physics], 6 * s.n ** 3, bb.np3(s.N)), generator=gen,
                          dtype=torch.float64).numpy() * 1e-2 for s in specs]
    B = BatchSolver(specs, dtype=torch.float64, states=states)
    q0 = [q.clone() for q in B.q]
    for s, (_, _, _, tile) in zip(specs, kinds):
        if tile:
            B.set_tile(s.physics, s.N, tile)
    for n in (1, 2):
        B.run(n, graph=graph)
    torch.cuda.synchronize()
    for p, spec in enumerate(specs):
        s = bb.DGSolver(B.meshes[p], spec.N, spec.physics, dtype=torch.float64, tau=spec.tau)
        s.set_tile(B.tile(spec.physics, spec.N), 256)
        q, r = q0[p].clone(), torch.zeros_like(q0[p])
        s.run(q, r, B.dt(p), 3, graph=False)
        torch.cuda.synchronize()
        assert torch.equal(q, B.q[p]) and torch.equal(r, B.res[p]), p
