"""The mixed policy keeps its cells and faces in an order of its own on the device (a Hilbert curve,
sorted in blocks of 2048); everything that crosses the boundary is in the caller's.  At sizes around
the blocks of that sort: an uploaded state comes back in place (to float), and one stage's outputs
agree, entry by entry, with those of the fp64 policy, which keeps the caller's order (FP32 arithmetic:
1e-4 of each array's scale, far below the differences between entries of the fields used)."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 3), (45, 45), (64, 32), (683, 3), (70, 59)])
def test_arrays_cross_the_boundary_in_the_callers_order(nx, ny):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, CudaSolver, mesh as M, precompute

    if not gpu_available():
        pytest.skip("no CUDA device")
    m = M.quad_grid(nx, ny)
    c = m.cell_centres()
    W = np.stack([2.0 + c[:, 0] + 0.3 * c[:, 1], 0.5 * c[:, 0] - 0.2, 0.4 * c[:, 1] + 0.1 * c[:, 0],
                  1.5 + 0.5 * c[:, 0] * c[:, 1] + 0.2 * c[:, 1]], axis=1)
    cfg = CaseConfig(stencilType="edgeNeighbour")
    hf = precompute(m, cfg, W, W[m.owner[m.n_internal_faces:]], want_rbf64=True)
    s, r = (CudaSolver(hf, cfg, policy=p) for p in ("mixed", "fp64"))
    a, b = s.stage_debug(0, 1e-6), r.stage_debug(0, 1e-6)
    for f in ("faceFD", "gradFD", "Flux", "FD", "cFD"):
        scale = np.abs(b[f]).max(axis=0) + 1e-30 if b[f].size else 1.0
        assert (np.abs(a[f] - b[f]) <= 1e-4 * scale.max()).all() if b[f].size else a[f].size == 0, f
    rng = np.random.default_rng(3)
    fd, u = 1.0 + rng.random(hf.FD.shape), 1.0 + rng.random(hf.cFD.shape)
    s.upload_state(FD=fd, cFD=u, cFDold=u)
    out = s.state()
    assert np.array_equal(out["FD"], fd.astype(np.float32).astype(np.float64))
    assert np.abs(out["cFD"] - u).max() <= 2.0 ** -46 * np.abs(u).max()
    s.close()
    r.close()
