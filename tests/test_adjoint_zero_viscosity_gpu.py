"""The viscosity contraction of the adjoint, lambda^T dR/d eta, where the residual is linear in eta: it does not
depend on eta at all, so it has to be the same numbers for every viscosity, cells of zero viscosity
included, and so do the transposed rows of a state whose viscosity is zero everywhere (finite: no quotient
by eta enters).

Tolerance: none.  The contraction is formed from lambda, the metric and the strain rates only.
"""
import numpy as np
import pytest

import sphericalstokes_gb300 as S
from sphericalstokes_gb300 import adjoint as A

pytestmark = pytest.mark.gpu

FIELDS = ("V1", "V2", "V3", "P")
CASES = [("spherical", dict(bc="stress", sig_bc=(0.0, 0.5, -0.5)), (13, 11, 9)), ("spherical", dict(bc="diapir"), (5, 34, 6)),
         ("cylindrical", dict(bc="stress", sig_bc=(0.0, 0.3, -0.3)), (11, 9, 10)), ("cartesian", dict(bc="diapir"), (10, 5, 9))]


@pytest.mark.parametrize("geom,kw,n", CASES)
@pytest.mark.parametrize("interior", [False, True])
def test_contraction_does_not_depend_on_the_viscosity(geom, kw, n, interior):
    rng = np.random.default_rng(3)
    if geom == "spherical" and kw["bc"] == "stress":
        p = S.sector_params(n, rheology="linear", **kw)
    else:
        p = S.default_params(geom, n1=n[0], n2=n[1], n3=n[2], rheology="linear", **kw)
    with S.Solver(p) as sv:
        for f in FIELDS:
            sv.set(f, rng.standard_normal(sv.dims(f)))
        lam = {f: rng.standard_normal(sv.dims(f)) for f in FIELDS}

        def contraction(eta):
            sv.set("ETA", eta)
            g = A.vjp(sv, lam, interior=interior)
            assert all(np.all(np.isfinite(a)) for a in g.values())
            return g["ETA"]
        want = contraction(np.ones(n))
        assert np.count_nonzero(want) == want.size - 8  # (the eight corner cells enter no momentum row)
        eta = np.exp(2 * rng.standard_normal(n))
        np.testing.assert_array_equal(contraction(eta), want)
        np.testing.assert_array_equal(contraction(1e-200 * eta), want)
        holes = np.where(rng.random(n) < 0.3, 0.0, eta)
        holes[1:4, :, :2] = 0.0  # whole edges among them
        np.testing.assert_array_equal(contraction(holes), want)
        np.testing.assert_array_equal(contraction(np.zeros(n)), want)
