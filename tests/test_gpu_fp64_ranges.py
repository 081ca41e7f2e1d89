"""The fp64 policy's kernels where their integer comparisons, FP32-seeded reciprocals and roots and
the FP32 look at the entropy fix could go wrong: SI units (large products of temperatures), small
units, a transonic expansion (the fix is active), and meshes at the edges of the small blocks, each
against the FP64 oracle, stage by stage over two steps.  1e-10 and identical switches, the bounds of
the policy's other oracle tests: every kernel value is a few ulps from the oracle's."""
import numpy as np
import pytest

from conftest import gpu_available, rel_err

pytestmark = pytest.mark.gpu

FIELDS = ["faceFD", "gradFD", "Flux", "Res", "FD", "cFD"]


def _case(kind):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, mesh as M

    cfg = CaseConfig(stencilType="edgeNeighbour", CFL=0.3)
    if kind in ("si", "small"):
        R = 287.0 if kind == "si" else 1e-3
        m = M.riemann_mixed(14, seed=2)
        W, Wb = M.riemann_fields(m)
        p, T = (1e5, 300.0) if kind == "si" else (1e-2, 5.0)
        u = np.sqrt(R * T / M.R_GAS)  # the same Mach numbers
        scale = np.array([p, u, u, T])
        return m, W * scale, Wb * scale, CaseConfig(R=R, Cv=2.5 * R, stencilType="edgeNeighbour", CFL=0.3)
    if kind == "sonic":
        m = M.quad_grid(40, 3)
        x = m.cell_centres()[:, 0]
        W = np.stack([1.0 + 0.2 * np.sin(9.0 * x), 0.6 + 0.9 * x, 0.05 * np.cos(5.0 * x), 1.0 + 0.1 * np.cos(7.0 * x)], 1)
        return m, W, W[m.owner[m.n_internal_faces:]], cfg
    nx, ny = kind
    m = M.quad_grid(nx, ny)
    c = m.cell_centres()
    W = np.stack([1.0 + 0.3 * np.sin(8.0 * c[:, 0] + 3.0 * c[:, 1]), 0.4 * np.cos(6.0 * c[:, 0]),
                  0.3 * np.sin(5.0 * c[:, 1] + 1.0), 1.0 + 0.2 * np.cos(9.0 * c[:, 0] - c[:, 1])], 1)
    return m, W, W[m.owner[m.n_internal_faces:]], cfg


@pytest.mark.parametrize("kind", ["si", "small", "sonic", (31, 1), (32, 1), (33, 1), (11, 12)], ids=str)
def test_fp64_stages_match_the_oracle(kind):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CudaSolver, precompute
    from oracle.oracle import Oracle

    if not gpu_available():
        pytest.skip("no CUDA device")
    m, W, Wb, cfg = _case(kind)
    hf = precompute(m, cfg, W, Wb, want_rbf64=True)
    s = CudaSolver(hf, cfg, policy="fp64")
    o = Oracle(hf, cfg.R, cfg.Cv, "fp64")
    st = o.new_state()
    for step in range(2):
        dt = o.delta_t(st["FD"], cfg.CFL)
        assert s.set_delta_t() == pytest.approx(dt, rel=1e-13)
        for k in range(3):
            a = s.stage_debug(k, dt)
            c = o.stage(st, k, dt)
            assert np.array_equal(a["shockIndicator"], c["shockIndicator"]), f"flags differ step {step} stage {k}"
            for f in FIELDS:
                if f == "Res":  # a sum of fluxes: against their scale
                    assert np.abs(a[f] - c[f]).max() <= 1e-10 * np.abs(c["Flux"]).max(), (f, step, k)
                else:
                    assert rel_err(a[f], c[f]) <= 1e-10, (f, step, k)
            s.upload_state(FD=c["FD"], cFD=c["cFD"], cFDold=c["cFD"] if k == 2 else None)
    s.close()
