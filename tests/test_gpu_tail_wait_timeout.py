"""The bounded waits of the fused stage's two kernels, one by one: a wait that runs out marks the
solver's error word and the call reports AFAR_ERR_CUDA, also where the copy lands just after the wait gave
up; the context stays usable and the next steps are those of an untouched solver.  The waits run out
through the library's test hook (bytes that are never issued, a limit of 2^20 clocks)."""
import numpy as np
import pytest

from conftest import gpu_available, small_cases

pytestmark = pytest.mark.gpu

RECONSTRUCT_ROWS, TAIL_FACES, TAIL_STATES = 1, 2, 3


@pytest.mark.parametrize("case", ["mixed_riemann", "ffs_tri"])
@pytest.mark.parametrize("where,late", [(RECONSTRUCT_ROWS, 0), (TAIL_FACES, 0), (TAIL_FACES, 1), (TAIL_STATES, 0)])
def test_each_wait_that_runs_out_is_reported(case, where, late):
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import AfarError, CaseConfig, CudaSolver, _ffi, precompute

    m, W, Wb, st = small_cases()[case]
    cfg = CaseConfig(stencilType=st)
    hf = precompute(m, cfg, W, Wb)
    L = _ffi.lib()
    s, ref = CudaSolver(hf, cfg, policy="mixed"), CudaSolver(hf, cfg, policy="mixed")
    for v in (s, ref):
        v.set_tuning(0)  # the tile-staged reconstruct; the last tile of both meshes has lanes without a cell
    _ffi.check(L.afar_debug_wait_injection_at(0, where, 16, late, 1 << 20))
    try:
        with pytest.raises(AfarError) as err:
            s.run(1, dt=1e-4)
    finally:
        _ffi.check(L.afar_debug_wait_injection(0, 0, 0))
    assert err.value.status == 4  # AFAR_ERR_CUDA
    assert "timed out" in str(err.value) and "state is not valid" in str(err.value)
    s.upload_state(FD=hf.FD, cFD=hf.cFD, cFDold=hf.cFD)
    for v in (s, ref):
        v.run(3, dt=1e-4)
    assert all(np.array_equal(s.state()[f], ref.state()[f]) for f in ("FD", "cFD", "shockIndicator"))
    s.close()
    ref.close()


def test_unknown_waits_are_refused():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import _ffi

    L = _ffi.lib()
    assert L.afar_debug_wait_injection_at(0, 4, 16, 0, 1 << 20) == 1
    assert L.afar_debug_wait_injection_at(0, -1, 16, 0, 1 << 20) == 1
    assert L.afar_debug_wait_injection_at(0, TAIL_STATES, 16, 1, 1 << 20) == 1
