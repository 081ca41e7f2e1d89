"""The mixed policy's fused step leaves the last stage's limiter untransformed, and a Courant step alone
(set_delta_t) its switch types undecided, until they are asked for.  What they are worked out from must be
the state and the intermediates of that stage, whatever call replaces those in between: flags and limiters
are the ones that a twin reads straight away."""
import ctypes as C

import numpy as np
import pytest

from conftest import gpu_available, small_cases

pytestmark = pytest.mark.gpu


def bundle(face_neighbour=False):
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, mesh as M, precompute

    if face_neighbour:
        m = M.quad_grid(101, 97, 0.0, 1.2, 0.0, 1.0)
        W, Wb = M.riemann_fields(m)
        cfg = CaseConfig(stencilType="faceNeighbour", CFL=0.2)
    else:
        m, W, Wb, st = small_cases()["mixed_riemann"]
        cfg = CaseConfig(stencilType=st, CFL=0.2)
    return precompute(m, cfg, W, Wb), cfg


def switches(s):
    return s.state()["shockIndicator"], s.switch_counts(), s.limiter64()


@pytest.mark.parametrize("replace", ["upload", "restore"])
def test_a_replaced_state_keeps_the_head_s_switches(replace):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CudaSolver

    hf, cfg = bundle()
    s, twin = (CudaSolver(hf, cfg, policy="mixed") for _ in range(2))
    for v in (s, twin):
        v.save()
        v.run(12)
        v.set_delta_t()
    if replace == "upload":
        x = hf.FD.copy()
        x[:, 0] *= 1.0 + 0.5 * np.sin(np.arange(x.shape[0]))
        x[:, 3] *= 1.0 + 0.4 * np.cos(3.0 * np.arange(x.shape[0]))
        s.upload_state(FD=x)
    else:
        s.restore()
    (a, ca, la), (b, cb, lb) = switches(s), switches(twin)
    assert np.array_equal(a, b)
    assert ca == cb
    assert np.array_equal(la, lb)
    assert np.abs(a).any() and len(np.unique(lb)) > 2  # there is something to get wrong
    s.close()
    twin.close()


def test_the_tuner_s_launches_leave_the_switches():
    from afar_cudaeuler2dmixo3rk3solver_gb300 import _ffi
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CudaSolver

    hf, cfg = bundle(face_neighbour=True)
    L = _ffi.lib()
    # a variant asked for before the upload, so that this mesh class has not been timed yet when it is dropped
    s = CudaSolver.__new__(CudaSolver)
    s.cfg, s.fields, s.policy, s.h, z = cfg, hf, "mixed", C.c_void_p(), hf.sizes
    _ffi.check(L.afar_solver_create(C.byref(s.h), _ffi.POLICIES["mixed"], 0))
    _ffi.check(L.afar_set_tuning(s.h, 0))
    s._fp = hf.to_c()
    _ffi.check(L.afar_setDeviceFieldData(s.h, C.byref(s._fp), z["cellsNum"], z["facesNum"], z["totalBoundaryFacesNum"]))
    _ffi.check(L.afar_setDeviceFieldDataStencil(
        s.h, C.byref(s._fp), z["cellsNum"], z["facesNum"], z["patchesNum"], z["totalBoundaryFacesNum"],
        z["maxStencilSize"], z["maxCompactStencilSize"], z["maxLocalBlockStencilSize"],
        z["maxCompactLocalBlockStencilSize"]))
    _ffi.check(L.afar_set_gas(s.h, cfg.R, cfg.Cv))
    s.run(12)
    before = s.state()["shockIndicator"][1::2]
    s.set_tuning(-1)
    s.limiter64()
    assert np.array_equal(s.state()["shockIndicator"][1::2], before)
    assert before.any()
    twin = CudaSolver(hf, cfg, policy="mixed")
    for v in (s, twin):  # nor do they leave a Courant step
        v.upload_state(FD=hf.FD, cFD=hf.cFD, cFDold=hf.cFD)
        v.run(1)
    assert s.time()[1] == twin.time()[1]
    s.close()
    twin.close()


def test_a_batch_s_timing_leaves_no_switch_pending():
    """The timing of a batch's separate kernels decides its members' switches anew, of the state they have:
    reading a limiter afterwards does not mix those of the last stage in."""
    from afar_cudaeuler2dmixo3rk3solver_gb300 import Batch, CudaSolver

    hf, cfg = bundle()
    solvers = [CudaSolver(hf, cfg, policy="mixed") for _ in range(17)]
    solvers[0].set_tuning(1)  # one member's register pass: the batch runs, and times, the separate kernels
    batch = Batch("mixed")
    for s in solvers:
        s.run(12)
        batch.add(s)
    batch.schedule()
    after = solvers[1].state()["shockIndicator"]
    for s in solvers[1:]:
        s.limiter64()
        assert np.array_equal(s.state()["shockIndicator"], after)
    assert after.any()
    batch.close()
    for s in solvers:
        s.close()
