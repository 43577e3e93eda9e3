"""Correction sweeps by three kernels of their own: the TMA sweep (two points per thread in paired arithmetic), the cp.async
sweep, and one kernel per reference step.  (test_sweep_two_points_per_thread_equals_one of test_parity_gpu.py switches
between kernels that are one now.)

Bound 1e-5 of a field's largest value: the kernels evaluate the same sums in different orders, a rounding of 6e-8 or so
each, and the iteration damps what 57 sweeps add up.
"""
import pytest

import sphericalstokes_gb300 as S
from test_parity_gpu import X2_CASES, _params, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("other", ["cp_async", "simple"])
@pytest.mark.parametrize("geom,n,kw", X2_CASES)
def test_correction_sweeps_agree(monkeypatch, geom, n, kw, other):
    out = []
    for which in ("tma", other):
        monkeypatch.setenv("SPH_NO_TMA", "1" if which == "cp_async" else "0")
        nn = (n, n, n) if isinstance(n, int) else n
        p = _params(geom, nn, precision="mixed", kernels="simple" if which == "simple" else "auto", **kw)
        with S.Solver(p) as sv:
            sv.sweep(57)
            sv.sweep_apply()
            out.append({f: sv.get(f) for f in ("V1", "V2", "V3", "P")})
    for f in out[0]:
        assert relerr(out[1][f], out[0][f]) < 1e-5, f
