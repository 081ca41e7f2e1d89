"""The Courant step is the smallest over the faces of the state at hand: a step size worked out by
set_delta_t and then not used leaves nothing behind, whatever steps the solver next."""
import numpy as np
import pytest

from conftest import gpu_available, small_cases

pytestmark = pytest.mark.gpu


def bundle():
    if not gpu_available():
        pytest.skip("no CUDA device")
    from afar_cudaeuler2dmixo3rk3solver_gb300 import CaseConfig, precompute

    m, W, Wb, st = small_cases()["mixed_riemann"]
    cfg = CaseConfig(stencilType=st, CFL=0.1)
    return precompute(m, cfg, W, Wb, want_rbf64=True), cfg


@pytest.mark.parametrize("how", ["run", "run_timed", "profile_step", "save_restore", "upload", "batch"])
@pytest.mark.parametrize("policy", ["mixed", "fp64", "ref"])
def test_an_unused_courant_step_is_forgotten(policy, how):
    from afar_cudaeuler2dmixo3rk3solver_gb300 import Batch, CudaSolver

    if policy == "ref" and how == "batch":
        pytest.skip("the ref policy has no batches")
    hf, cfg = bundle()
    s, fresh = (CudaSolver(hf, cfg, policy=policy) for _ in range(2))
    s.set_delta_t()  # at 0.1: half of what follows
    if how == "save_restore":
        s.save()
        s.restore()
    if how == "upload":  # the same flow, as if replaced
        s.upload_state(FD=hf.FD, cFD=hf.cFD, cFDold=hf.cFD)
    for v in (s, fresh):
        if how == "batch":
            v.set_step_params(cfl=0.2)
            b = Batch(policy)
            b.add(v)
            b.run(1)
            b.close()
        elif how in ("run_timed", "profile_step"):
            getattr(v, how)(*([1] if how == "run_timed" else []), cfl=0.2)
        else:
            v.run(1, cfl=0.2)
    assert s.time()[1] == fresh.time()[1]
    assert np.array_equal(s.state()["cFD"], fresh.state()["cFD"])
    s.close()
    fresh.close()
