"""Device memory of a mixed solver: no more than that of the separate stage kernels' arrays alone (the
device order, the state's further buffers and the fused stage's lists take the place of arrays that the
fused stage does not use), and what shares a buffer keeps its values between the calls that need them."""
import numpy as np
import pytest

from conftest import gpu_available, small_cases

pytestmark = pytest.mark.gpu


def separate_bytes(z):
    """The arrays of a mixed solver that runs the separate kernels in the caller's order."""
    nc, nf, nb = z["cellsNum"], z["facesNum"], z["totalBoundaryFacesNum"]
    S, M, ldc = z["maxStencilSize"], z["maxCompactStencilSize"], (nc + 31) // 32 * 32
    state = (16 + 16 + 2) * (nc + nb) + 64 * nc + 32 * (nc + nb)  # centres, W, flags; U, Un; transfers
    cells = 20 * nc + 48 * nc + 32 * nc + 2 * nc  # volumes and reciprocals; gradients, limiters; residual; counts
    faces = 40 * (nf + nb) + 32 * nf + 16 * (nf + nb) + 24 * nf + 16 * nb + 8 * nf + 5 * nb + 16 * nf + 16 * (nf + nb)
    rows = (4 * S + 4 * M + 24 * M + 4 * M * (S + 1)) * ldc
    return state + cells + faces + rows


@pytest.mark.parametrize("name", ["quads", "quads_face", "triangles", "both"])
def test_no_more_memory_than_the_separate_kernels(name):
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, CudaSolver, mesh as M, precompute

    m = {"quads": lambda: M.quad_grid(137, 137), "quads_face": lambda: M.quad_grid(211, 160),
         "triangles": lambda: M.forward_step_triangles(20_000, seed=2), "both": lambda: M.riemann_mixed(150, seed=3)}[name]()
    W, Wb = M.uniform_fields(m, 1.0, 0.5, 0.0, 1.0)
    cfg = CaseConfig(stencilType="faceNeighbour" if name == "quads_face" else "edgeNeighbour")
    hf = precompute(m, cfg, W, Wb, device=0)
    s = CudaSolver(hf, cfg, policy="mixed")
    assert s.device_bytes() <= separate_bytes(hf.sizes) + 65536  # the ends of 40 arrays, the tensor maps
    s.close()


@pytest.mark.parametrize("kind", ["fused", "gauss", "separate"])
def test_fields_read_inside_a_step_do_not_change_it(kind):
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import Batch, CaseConfig, CudaSolver, precompute

    m, W, Wb, st = small_cases()["mixed_riemann"]
    cfg = CaseConfig(stencilType=st, CFL=0.2)
    hf = precompute(m, cfg, W, Wb, gauss_flux=kind == "gauss")
    if kind == "separate":  # a stencil that does not start with the cells across the faces
        S = hf.sizes["maxStencilSize"]
        ls = hf.a["localStencil"].reshape(-1, S)
        ls[5, [0, 1]] = ls[5, [1, 0]]
    a, b = (CudaSolver(hf, cfg, policy="mixed", gauss_flux=kind == "gauss") for _ in range(2))
    for _ in range(3):
        dt = a.set_delta_t()
        assert b.set_delta_t() == dt
        a.write_field()
        a.state()
        a.evolve(dt)
        b.evolve(dt)
        assert all(np.array_equal(a.state()[f], b.state()[f]) for f in ("FD", "cFD", "shockIndicator"))
    if kind != "gauss":  # the separate kernels of a batch, read between its runs
        out = []
        for v, read in ((a, True), (b, False)):
            batch = Batch("mixed")
            batch.add(v)
            v.set_step_params()
            batch.set_schedule(64, 256)
            for _ in range(2):
                batch.run(1)
                if read:
                    v.state()
            batch.close()
            out.append(v.state()["cFD"])
        assert np.array_equal(*out)
    if kind == "gauss":  # and back to the face-centre flux
        for v in (a, b):
            v.set_face_gauss_flux(None)
            v.run(2, dt=1e-4)
        x, y = a.stage_debug(0, 1e-4), b.stage_debug(0, 1e-4)
        assert all(np.array_equal(x[f], y[f]) for f in ("Flux", "Res", "cFD"))
    a.close()
    b.close()


def test_a_restored_snapshot_brings_its_fixed_ghosts():
    """Ghosts that keep their uploaded state are in each of the state's buffers: a restored snapshot's are the
    ones it was taken with, whatever was uploaded since, and an upload's its own."""
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, CudaSolver, precompute

    m, W, Wb, st = small_cases()["corner_flow"]
    cfg = CaseConfig(R=0.7142857, Cv=1.7857142857, CFL=0.08, stencilType=st, cOrder=7, fOrder=5)
    hf = precompute(m, cfg, W, Wb)
    other = hf.FD.copy()
    other[hf.nc:, 0] *= 0.5  # another inlet
    up = {"a": dict(FD=hf.FD, cFD=hf.cFD, cFDold=hf.cFD), "b": dict(FD=other, cFD=hf.cFD, cFDold=hf.cFD)}
    want = {}
    for k, u in up.items():
        s = CudaSolver(hf, cfg, policy="mixed")
        s.upload_state(**u)
        s.run(4, dt=1e-4)
        want[k] = s.state()["FD"]
        s.close()
    assert not np.array_equal(want["a"], want["b"])
    s = CudaSolver(hf, cfg, policy="mixed")

    def steps(k):
        s.run(4, dt=1e-4)
        assert np.array_equal(s.state()["FD"], want[k])

    s.save()
    steps("a")
    s.upload_state(**up["b"])
    steps("b")
    s.restore()
    steps("a")
    s.restore()
    steps("a")
    s.upload_state(**up["b"])
    s.save()
    s.upload_state(**up["a"])
    s.restore()
    steps("b")
    s.restore()
    steps("b")
    s.upload_state(**up["a"])
    steps("a")
    s.close()
