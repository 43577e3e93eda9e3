"""A run of iterations computes the smoothed viscosity of each but its first together with the
boundary values of the one before; one iteration at a time computes it by itself.  Same integer maxima,
same arithmetic otherwise: equal bits in every field, at grids around the warp width and the smallest."""
import numpy as np
import pytest

import sphericalstokes_gb300 as S

pytestmark = pytest.mark.gpu

FIELDS = ("P", "V1", "V2", "V3", "TAU11", "TAU22", "TAU33", "TAU12", "TAU13", "TAU23", "ETA", "ETA_SM", "DT_R")
KINDS = [
    ("spherical", dict(bc="diapir", rheology="tau_power", n_exp=3.0)),
    ("spherical", dict(bc="stress", rheology="edot_power_relax", n_exp=3.0, relax=0.5, edot_bg=0.25, sig_bc=(0.0, 0.5, -0.5))),
    ("spherical", dict(bc="free_slip", rheology="linear", etasm_passes=2)),
    ("cylindrical", dict(rheology="tau_power_relax", n_exp=2.0, relax=0.1)),
    ("cartesian", dict(rheology="tau_power_relax", n_exp=2.0, relax=0.1)),
]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [(5, 5, 5), (33, 7, 10), (40, 35, 6)])
@pytest.mark.parametrize("geometry,kw", KINDS)
def test_run_equals_single_iterations(geometry, kw, n, precision):
    p = S.default_params(geometry, n1=n[0], n2=n[1], n3=n[2], precision=precision, **kw)
    rng = np.random.default_rng(5)
    out = []
    eta = None
    for steps in ((6,), (1,) * 6):
        with S.Solver(p) as sv:
            if eta is None:
                eta = np.exp(rng.uniform(-1, 1, sv.dims("ETA")))
                v = {f: 1e-3 * rng.standard_normal(sv.dims(f)) for f in ("V1", "V2", "V3")}
            for f, a in list(v.items()) + [("ETA", eta), ("ETA_INI", eta), ("ETA_PL", eta)]:
                sv.set(f, a)
            for k in steps:
                sv.step(k)
            out.append({f: sv.get(f) for f in FIELDS})
    for f in FIELDS:
        np.testing.assert_array_equal(out[0][f], out[1][f], err_msg=f)
    assert np.isfinite(out[0]["V1"]).all() and np.abs(out[0]["V1"]).max() > 0.0
