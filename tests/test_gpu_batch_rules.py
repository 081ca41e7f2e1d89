"""Batches whose way of stepping is chosen by their members' numbers and sizes: chains of the fused stage side
by side (small members) and in turn (large ones), and the separate kernels for many small members with wide
stencils.  Each against the separate kernels with forced block sizes: the same bits."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu


# (members, quads a side, stencil): chains side by side; chains in turn; many small members; tiles of 96 cells
@pytest.mark.parametrize("members,n,stencil,launches", [(50, 33, "edgeNeighbour", 12), (50, 152, "faceNeighbour", 12),
                                                        (97, 24, "faceNeighbour", 13), (33, 61, "faceNeighbour", 13)],
                         ids=str)
def test_every_way_is_the_separate_kernels(members, n, stencil, launches):
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import Batch, CaseConfig, CudaSolver, mesh as M, precompute

    m = M.quad_grid(n, n, 0.0, 1.2, 0.0, 1.0)
    W, Wb = M.riemann_fields(m)
    cfg = CaseConfig(stencilType=stencil, CFL=0.2)
    hf = precompute(m, cfg, W, Wb, device=0)
    solvers = [CudaSolver(hf, cfg, policy="mixed") for _ in range(members)]
    assert solvers[0].step_launches() == 6 and solvers[0].launches_per_step() == 13
    out = []
    for schedule in ((0, 0), (128, 256)):
        batch = Batch("mixed")
        for i, s in enumerate(solvers):
            s.upload_state(FD=hf.FD, cFD=hf.cFD, cFDold=hf.cFD)
            s.set_time(0.0)
            s.set_step_params(cfl=0.1 + 0.001 * i)
            batch.add(s)
        assert batch.step_launches() == launches
        batch.set_schedule(*schedule)
        assert batch.step_launches() == (13 if schedule[0] else launches)
        batch.run(3)
        out.append([(s.state(), s.time()[0]) for s in solvers[:: max(1, members // 12)] + solvers[-1:]])
        batch.close()
    for (x, tx), (y, ty) in zip(*out):
        assert tx == ty
        assert all(np.array_equal(x[f], y[f]) for f in ("FD", "cFD", "shockIndicator"))
    for s in solvers:
        s.close()
