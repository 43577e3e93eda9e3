"""Device memory of the adjoint and of the advection step, and that neither leaves a trace in the state.

The workspace is at most 33 boxes of the padded grid in FP64 beside the state, for every call: a grid whose state and 33
boxes fit the device has an adjoint.  Boxes are (n1 + 1 rounded up to 32) x (n2 + 1) x (n3 + 1) doubles; one more
is the staging field of the host copies; allocations are rounded up to 2 MiB each.
"""
import numpy as np
import pytest

import sphericalstokes_gb300 as S
from sphericalstokes_gb300 import adjoint as A
from sphericalstokes_gb300 import ascent

pytestmark = pytest.mark.gpu

FIELDS = ("V1", "V2", "V3", "P")
STATE = FIELDS + ("TAU11", "TAU22", "TAU33", "TAU12", "TAU13", "TAU23", "ETA", "TII")
LAWS = {"linear": dict(rheology="linear"), "law": dict(rheology="edot_power_relax", n_exp=3.0, relax=0.5, edot_bg=0.25)}


def start(sv, seed=5):
    rng = np.random.default_rng(seed)
    for f in FIELDS:
        sv.set(f, 0.1 * rng.standard_normal(sv.dims(f)))
    if sv.params.precision == S.PREC["fp64"]:
        sv.apply_bc()


def adjoint_calls(sv, seed=6):
    rng = np.random.default_rng(seed)
    lam = {f: rng.standard_normal(sv.dims(f)) for f in FIELDS}
    g = A.vjp(sv, lam)
    gi, gn = A.law_vjp(sv)
    out, info = A.adjoint_solve(sv, lam, tol=1e-30, maxiter=9, nout=4)
    phi = [rng.standard_normal(sv.dims("P")) for _ in range(4)]
    new = ascent.advect(sv, phi, 1e-3, 1e-2)
    return [*g.values(), gi, np.array(gn), *out.values(), np.array(info.err), *new]


@pytest.mark.parametrize("law", LAWS)
def test_workspace(law):
    torch = pytest.importorskip("torch")
    n = (95, 63, 63)
    with S.Solver(S.sector_params((13, 11, 9), bc="stress", **LAWS[law])) as sv:  # (the kernels' modules are loaded)
        start(sv)
        adjoint_calls(sv)
    with S.Solver(S.sector_params(n, bc="stress", **LAWS[law])) as sv:
        start(sv)
        free = torch.cuda.mem_get_info()[0]
        adjoint_calls(sv)
        used = free - torch.cuda.mem_get_info()[0]
    box = 8 * ((n[0] + 1 + 31) // 32 * 32) * (n[1] + 1) * (n[2] + 1)
    assert 0 < used <= 34 * box + 2 * (2 << 20), used / box


@pytest.mark.parametrize("law", LAWS)
@pytest.mark.parametrize("bc", ["stress", "free_slip"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [(13, 11, 9), (33, 5, 7)])
def test_no_trace_in_the_state(law, bc, precision, n):
    """iterations, a residual and a solve after adjoint calls are those without them, bit for bit, and so are the
    results of adjoint calls after iterations and solves"""
    runs = []
    for between in (False, True):
        with S.Solver(S.sector_params(n, bc=bc, precision=precision, **LAWS[law])) as sv:
            start(sv)
            first = adjoint_calls(sv) if between else None
            state = []
            for _ in range(2):
                if precision == "fp64":
                    sv.step(3)
                else:
                    sv.solve(tol=1e-30, maxiter=20, nout=10, criterion="residual")
                if between:
                    adjoint_calls(sv)
                state += [*A.residual_fields(sv).values()] + [sv.get(f) for f in STATE]
            sv.solve(tol=1e-30, maxiter=20, nout=10, criterion="residual")
            state += [sv.get(f) for f in STATE]
            if between:
                start(sv)
                for f in ("ETA", "ETA_INI"):
                    sv.set(f, np.ones(n))
                again = adjoint_calls(sv)
                with S.Solver(sv.params) as fresh:
                    start(fresh)
                    for f in ("ETA", "ETA_INI"):
                        fresh.set(f, np.ones(n))
                    for x, y in zip(again, adjoint_calls(fresh)):
                        np.testing.assert_allclose(x, y, rtol=1e-9, atol=1e-9 * np.abs(y).max())  # (atomics of the stress ghosts)
        runs.append(state)
    for x, y in zip(*runs):
        np.testing.assert_array_equal(x, y)
