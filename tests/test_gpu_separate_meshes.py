"""Mixed meshes that keep the separate stage kernels: those whose faces are not in the lists of both
their cells as the fused stage needs it (a cell that names a face with the other sign, or whose stencil
does not start with the cells across its faces, in order), and those with tiles that reach more cells than
a tile's lists hold.  They are solved in the device's cell order all the same: whole steps are those of the
stages one by one, to the bit, and a stage's arrays are those of the fp64 policy, which keeps the
caller's order (FP32 arithmetic: 1e-4 of each array's scale, and in a gradient, a difference of
neighbours over their spacing, twice the FP32 spacing of the states over it)."""
import numpy as np
import pytest

from conftest import gpu_available

pytestmark = pytest.mark.gpu


def bundle(kind):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, mesh as M, precompute

    if not gpu_available():
        pytest.skip("no CUDA device")
    # long cells in columns of 400: a tile of 152 has all of two further columns' parts across its border
    m = M.quad_grid(30, 400, 0.0, 1.0, 0.0, 2e-4) if kind == "columns" else M.riemann_mixed(30, seed=5)
    c = m.cell_centres()
    c = (c - c.min(axis=0)) / (c.max(axis=0) - c.min(axis=0))
    W = np.stack([2.0 + 0.3 * np.sin(5 * c[:, 0]) + 0.2 * c[:, 1], 0.5 * c[:, 0] - 0.2, 0.1 * c[:, 0] + 0.05 * c[:, 1],
                  1.5 + 0.2 * np.cos(4 * c[:, 0]) + 0.1 * c[:, 1]], axis=1)
    cfg = CaseConfig(stencilType="edgeNeighbour")
    hf = precompute(m, cfg, W, W[m.owner[m.n_internal_faces:]], want_rbf64=True)
    M_, S = hf.sizes["maxCompactStencilSize"], hf.sizes["maxStencilSize"]
    cells = [c for c in range(7, hf.nc, 97) if hf.a["compactStencilSize"][c] >= 3]
    if kind == "signs":  # both cells of a face name it with the other sign
        cf = hf.a["cellFaces"].reshape(-1, M_)
        for c in cells:
            f = next(abs(int(x)) for x in cf[c, :hf.a["compactStencilSize"][c]] if abs(int(x)) <= hf.nf)
            cf[np.abs(cf) == f] *= -1
            for r in (hf.a["RBFbasis"], hf.a["RBFbasis64"]):  # each cell keeps its weights
                rows = r.reshape(hf.nf, 2, S + 1)
                rows[f - 1] = rows[f - 1, ::-1].copy()
    elif kind == "stencil":
        st = hf.a["localStencil"].reshape(-1, S)
        for c in cells:
            st[c, [0, 1]] = st[c, [1, 0]]
    return hf, cfg, 5e-7 if kind == "columns" else 1.0 / 60.0


@pytest.mark.parametrize("kind", ["signs", "stencil", "columns"])
def test_meshes_without_the_fused_stage(kind):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CudaSolver

    hf, cfg, spacing = bundle(kind)
    a, b, r = CudaSolver(hf, cfg, policy="mixed"), CudaSolver(hf, cfg, policy="mixed"), CudaSolver(hf, cfg, policy="fp64")
    dt = 1e-9 if kind == "columns" else 1e-5
    a.save()
    assert a.profile_step(dt=dt)["bvd"] > 0.0  # the separate kernels run
    a.restore()
    for step in range(2):
        a.run(1, dt=dt)
        for k in range(3):
            x, y = b.stage_debug(k, dt), r.stage_debug(k, dt)
            if step == 0 and k == 0:
                for f in ("faceFD", "gradFD", "Flux", "FD", "cFD"):
                    assert np.isfinite(y[f]).all(), f
                    rounding = 2.0 ** -22 * np.abs(hf.FD).max() / spacing if f == "gradFD" else 0.0
                    assert (np.abs(x[f] - y[f]) <= 1e-4 * np.abs(y[f]).max() + rounding).all(), f
        u, v = a.state(), b.state()
        for f in ("FD", "cFD", "shockIndicator"):
            assert np.array_equal(u[f], v[f]), (step, f)
    assert np.array_equal(a.limiter64(), b.limiter64())
    for s in (a, b, r):
        s.close()
