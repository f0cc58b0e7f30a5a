"""The FP64 stage kernel's two tile forms (whole lift stacks in shared memory, and the
face-by-face lift where they do not fit) over degrees, tile sizes and remainders."""
import numpy as np
import pytest

from oracle import meshdata
from test_gpu_stage_any_count import mesh_with_lone_elements, rel

pytestmark = pytest.mark.gpu

CODE = {"wave": 0, "maxwell": 1, "advection": 2, "advection3": 3}


@pytest.mark.parametrize("physics", sorted(CODE))
@pytest.mark.parametrize("N", [1, 2, 8, 12, 15, 20])
def test_every_tile_matches_the_oracle(cuda, bb, oracle_cpu, physics, N):
    """The right-hand side at the default tile, one element per block and the largest tiles that
    shared memory takes (degree 12 and up: no whole stacks): the repository's FP64 tolerance,
    1e-12 per field."""
    import torch
    m = bb.uniform_tet_mesh(2)
    if (physics, N) == ("maxwell", 20):   # one element takes 288 KB of shared memory
        with pytest.raises(bb.BBError):
            bb.DGSolver(m, N, physics, dtype=torch.float64, tau=1.0)
        return
    s = bb.DGSolver(m, N, physics, dtype=torch.float64, tau=1.0)
    q = np.random.default_rng(N).uniform(-1, 1, (s.nf, m.K, s.Np))
    want = torch.tensor(oracle_cpu.rhs(CODE[physics], N, q, meshdata.build(m, N), tau=1.0),
                        device=cuda)
    qd = torch.tensor(q, device=cuda)
    tiles = [s.tile[0], 1, 2, 3, 5, 8, 12, 20]
    ran = 0
    for e in tiles:
        try:
            s.set_tile(e, 256)
        except bb.BBError:
            continue                     # exceeds shared memory
        ran += 1
        err = rel(s.rhs(qd), want)
        assert max(err) < 1e-12, (e, err)
    assert ran >= 2


@pytest.mark.parametrize("physics,N", [("wave", 3), ("maxwell", 7), ("advection", 5), ("wave", 13),
                                       ("maxwell", 13)])
@pytest.mark.parametrize("extra", [0, 1, 3])
def test_partial_last_tile_and_steps(cuda, bb, physics, N, extra):
    """Two LSRK steps at several tile sizes, K = 48 + extra: 1e-12 of one another per field."""
    import torch
    m = mesh_with_lone_elements(bb, 2, extra)
    s = bb.DGSolver(m, N, physics, dtype=torch.float64, tau=1.0)
    gen = torch.Generator(device=cuda).manual_seed(N)
    q0 = torch.rand((s.nf, m.K, s.Np), generator=gen, device=cuda, dtype=torch.float64) * 2 - 1
    out = []
    for e in (1, 2, 4, 7):
        try:
            s.set_tile(e, 256)
        except bb.BBError:
            continue
        q = q0.clone()
        s.run(q, torch.zeros_like(q), s.dt_cfl(), 2)
        s.check()
        out.append(q)
    assert len(out) >= 2
    for q in out[1:]:
        assert max(rel(q, out[0])) < 1e-12
