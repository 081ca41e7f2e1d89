"""The mixed step's fused stage (reconstruct, then one kernel over tiles of 96, 152 or 192 cells that works
out the switch types, the fluxes and the update of its cells, its border cells again) against the
separate kernels, which afar_stage_debug and a batch with block sizes of its own still run: the same
bits, at one cell, around one tile and two, over walls, corners and every stencil kind."""
import numpy as np
import pytest

from conftest import gpu_available, small_cases

pytestmark = pytest.mark.gpu

FIELDS = ("FD", "cFD", "shockIndicator")


def case(name):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, mesh as M

    if not gpu_available():
        pytest.skip("no CUDA device")
    if name in ("corner_flow", "ffs_tri", "mixed_riemann"):
        m, W, Wb, st = small_cases()[name]
        if name == "corner_flow":
            return m, W, Wb, CaseConfig(R=0.7142857, Cv=1.7857142857, CFL=0.08, stencilType=st, cOrder=7, fOrder=5)
        return m, W, Wb, CaseConfig(stencilType=st, CFL=0.2)
    kind, a, b = name
    m = M.quad_grid(a, b) if kind == "quads" else M.forward_step_triangles(a, seed=b)
    c = m.cell_centres()
    W, _ = M.uniform_fields(m, 1.0, 0.5, 0.2, 1.0)
    W[:, 0] *= np.where(np.sin(9 * c[:, 0] + 5 * c[:, 1]) > 0.3, 1.6, 1.0)  # jumps: both flux kinds
    return m, W, W[m.owner[m.n_internal_faces:]], CaseConfig(stencilType="edgeNeighbour", CFL=0.2)


# quads: one cell, around one tile of 96, a remainder, either side of the change to tiles of 152 (4096 cells);
# triangles: tiles of 192.  50,000 and 532,000 quads: the other ways its launches follow one another
@pytest.mark.parametrize("name", [("quads", 1, 1), ("quads", 95, 1), ("quads", 12, 8), ("quads", 97, 1), ("quads", 61, 5),
                                  ("quads", 64, 64), ("quads", 241, 17), ("quads", 250, 200), ("quads", 760, 700), ("triangles", 5000, 2), "corner_flow",
                                  "ffs_tri", "mixed_riemann"], ids=str)
def test_fused_run_is_the_separate_kernels(name):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import Batch, CudaSolver, precompute

    m, W, Wb, cfg = case(name)
    hf = precompute(m, cfg, W, Wb, device=0)
    a, b, c = (CudaSolver(hf, cfg, policy="mixed") for _ in range(3))
    for step in range(3):
        a.run(1)
        dt = a.time()[1]
        if step == 0:  # the separate kernels' Courant step
            batch = Batch("mixed")
            batch.add(c)
            batch.set_schedule(128, 256)
            c.set_step_params()
            batch.run(1)
            assert c.time()[1] == dt
            batch.close()
        for k in range(3):
            b.stage_debug(k, dt)
        assert np.array_equal(a.limiter64(), b.limiter64())
        x, y = a.state(), b.state()
        for f in FIELDS:
            assert np.array_equal(x[f], y[f], equal_nan=True), (step, f)
    # the head alone leaves its stage's switch types, and the step that completes it, or does not, is the same
    t = a.time()[0]
    dt = a.set_delta_t()
    a.limiter64()
    b.stage_debug(0, dt)
    assert np.array_equal(a.state()["shockIndicator"], b.state()["shockIndicator"])
    for k in range(1, 3):
        b.stage_debug(k, dt)
    a.evolve(dt)
    assert all(np.array_equal(a.state()[f], b.state()[f], equal_nan=True) for f in FIELDS)
    # past t_end nothing moves; a restored state gives the same step again
    x = a.state()
    a.save()
    a.run(2, t_end=a.time()[0])
    assert all(np.array_equal(a.state()[f], x[f], equal_nan=True) for f in FIELDS[:2])
    a.run(2, dt=dt)
    y = a.state()
    a.restore()
    a.run(2, dt=dt)
    assert all(np.array_equal(a.state()[f], y[f], equal_nan=True) for f in FIELDS)
    assert a.time()[0] > t
    for s in (a, b, c):
        s.close()


# more members than one launch's parameters hold; cells of three and four faces together; 380 to 608 blocks of quads
@pytest.mark.parametrize("members,names", [(3, None), (48, None), (49, None), (6, [("quads", 100, 100)])], ids=str)
def test_fused_batch_is_the_separate_kernels(members, names):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import Batch, CudaSolver, precompute

    hfs = []
    for name in names or ("ffs_tri", "mixed_riemann", ("quads", 17, 9)):
        m, W, Wb, cfg = case(name)
        hfs.append((precompute(m, cfg, W, Wb), cfg))
    out = []
    for schedule in ((0, 0), (128, 256)):
        solvers = [CudaSolver(*hfs[i % len(hfs)], policy="mixed") for i in range(members)]
        batch = Batch("mixed")
        for i, s in enumerate(solvers):
            s.set_step_params(cfl=0.1 + 0.002 * i)
            batch.add(s)
        batch.set_schedule(*schedule)
        batch.run(3)
        out.append([(s.state(), s.time(), s.limiter64()) for s in solvers])
        batch.close()
        for s in solvers:
            s.close()
    for i, ((x, tx, lx), (y, ty, ly)) in enumerate(zip(*out)):
        assert tx == ty and np.array_equal(lx, ly), i
        assert all(np.array_equal(x[f], y[f], equal_nan=True) for f in FIELDS), i
