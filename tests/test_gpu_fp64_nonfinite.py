"""The fp64 policy's limiter forms a cell's four ratios with one reciprocal: a variable that is not finite in a
neighbour must not take the other three with it.  Cells with infinite entries: the switches of the first stage
are the FP64 oracle's, and a limiter that the oracle finds finite is finite."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("column,value", [(0, np.inf), (1, np.inf), (2, -np.inf)])
def test_infinite_neighbours(column, value):
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, CudaSolver, mesh as M, precompute
    from oracle.oracle import Oracle

    m = M.riemann_mixed(30, seed=5)
    W, Wb = M.riemann_fields(m)
    cfg = CaseConfig(stencilType="edgeNeighbour", CFL=0.2)
    hf = precompute(m, cfg, W, Wb, want_rbf64=True)
    cells = np.random.default_rng(0).choice(m.n_cells, 6, replace=False)
    hf.a["FD"][cells, column] = value
    o = Oracle(hf, cfg.R, cfg.Cv, "fp64")
    with np.errstate(all="ignore"):
        c = o.stage(o.new_state(), 0, 1e-4)
    s = CudaSolver(hf, cfg, policy="fp64")
    a = s.stage_debug(0, 1e-4)
    assert np.array_equal(a["shockIndicator"], c["shockIndicator"])
    assert np.isfinite(a["limiter"])[np.isfinite(c["limiter"])].all()
    s.close()
