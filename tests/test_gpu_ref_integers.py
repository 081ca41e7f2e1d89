"""The ref policy's conversions, selections and divisions off the FP64 pipe at the ends of their ranges,
against the ref oracle with the bounds its other tests have (face values and gradients 1e-12, the float
dissipation 1e-5 of the flux): velocities of zero, subnormal as float, subnormal as double.  And the
Courant step of both FP64 policies, evaluated only where FP32 bounds leave a face in question: 1e-13 of
the oracle's where the bounds are widest (a flow at Mach 1e5 along the faces) and where all faces tie."""
import numpy as np
import pytest

from conftest import gpu_available, rel_err

pytestmark = pytest.mark.gpu


def _solvers(W, m, policy):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, CudaSolver, precompute
    from oracle.oracle import Oracle

    cfg = CaseConfig(stencilType="edgeNeighbour", CFL=0.2)
    hf = precompute(m, cfg, W, W[m.owner[m.n_internal_faces:]], want_rbf64=True)
    s = CudaSolver(hf, cfg, policy=policy)
    mat = s.ls_matrix() if policy == "ref" else None
    return cfg, s, Oracle(hf, cfg.R, cfg.Cv, policy, **({"matrix32": mat} if mat is not None else {}))


@pytest.mark.parametrize("tiny", [0.0, 3e-42, 1e-310])
def test_ref_stage_with_tiny_velocities(tiny):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import mesh as M

    if not gpu_available():
        pytest.skip("no CUDA device")
    m = M.riemann_mixed(12, seed=6)
    c = m.cell_centres()
    W = np.stack([1.0 + 0.4 * np.sin(7.0 * c[:, 0]), tiny * np.cos(5.0 * c[:, 1]), -tiny * np.sin(3.0 * c[:, 0]),
                  1.0 + 0.2 * np.cos(6.0 * c[:, 1])], 1)
    cfg, s, o = _solvers(W, m, "ref")
    st = o.new_state()
    dt = o.delta_t(st["FD"], cfg.CFL)
    for k in range(3):
        a, b = s.stage_debug(k, dt), o.stage(st, k, dt)
        assert np.array_equal(a["shockIndicator"], b["shockIndicator"]), k
        for f in ("faceFD", "gradFD"):
            assert rel_err(a[f], b[f]) <= 1e-12, f
        assert np.abs(a["Flux"] - b["Flux"]).max() <= 1e-5 * np.abs(b["Flux"]).max()
        s.upload_state(FD=b["FD"], cFD=b["cFD"], cFDold=b["cFD"] if k == 2 else None)


@pytest.mark.parametrize("policy", ["ref", "fp64"])
@pytest.mark.parametrize("flow", ["fast", "cold", "uniform", "varied"])
def test_courant_step_is_the_smallest(policy, flow):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import mesh as M

    if not gpu_available():
        pytest.skip("no CUDA device")
    m = M.forward_step_triangles(1500, seed=8)
    c = m.cell_centres()
    W, _ = M.uniform_fields(m, 1.0, 3.0, 0.0, 1.0)
    if flow != "uniform":
        speed = {"fast": 1e5, "cold": 3.0, "varied": 3.0}[flow]
        angle = 3.0 * np.sin(4.0 * c[:, 0] + 5.0 * c[:, 1])
        W[:, 1], W[:, 2] = speed * np.cos(angle), speed * np.sin(angle)
        W[:, 3] = {"fast": 1.0, "cold": 1e-9, "varied": 1.0}[flow] * (1.0 + 0.5 * np.cos(6.0 * c[:, 0]))
    cfg, s, o = _solvers(W, m, policy)
    st = o.new_state()
    assert s.set_delta_t() == pytest.approx(o.delta_t(st["FD"], cfg.CFL), rel=1e-13)
    s.run(1)
    assert s.time()[1] == pytest.approx(o.delta_t(st["FD"], cfg.CFL), rel=1e-13)
