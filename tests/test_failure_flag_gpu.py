"""A bounded wait that runs out during FP32 iterations is reported by the call that ran them: the error word is set by
the wait self-test (a barrier that nothing completes, no copy in flight) and left for the next call."""
import pytest

import sphericalstokes_gb300 as S

pytestmark = pytest.mark.gpu

CALLS = {
    "step": ("fp32", lambda sv: sv.step(3)),
    "step_mixed": ("mixed", lambda sv: sv.step(3)),
    "solve_at_a_check": ("fp32", lambda sv: sv.solve(tol=1e-30, maxiter=20, nout=10, criterion="reference")),
    "solve_residual": ("fp32", lambda sv: sv.solve(tol=1e-30, maxiter=20, nout=10, criterion="residual")),
    "solve_between_checks": ("fp32", lambda sv: sv.solve(tol=1e-30, maxiter=7, nout=10, criterion="reference")),
    "warm_start": ("mixed", lambda sv: sv.solve(tol=1e-30, maxiter=40, nout=20, criterion="residual", warm_tol=1e-30, max_outer=0)),
}


@pytest.mark.parametrize("name", CALLS)
def test_time_out_is_reported(name):
    precision, call = CALLS[name]
    lib = S.load_library()
    with S.Solver(S.sector_params((15, 13, 11), bc="stress", rheology="linear", precision=precision)) as sv:
        call(sv)
        assert lib.sph_selftest_wait_flag(sv._h) == S.SPH_OK
        with pytest.raises(S.SphError, match="bounded wait"):
            call(sv)
        with pytest.raises(S.SphError, match="unusable"):
            call(sv)
