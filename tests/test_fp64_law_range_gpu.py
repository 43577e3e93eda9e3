"""The FP64 viscosity laws at the ends of the double range: a state at rest, strain rates and stresses whose
squared ratio to the law's scale leaves the range, cells without viscosity, an old and a target
viscosity whose product or quotient leaves it.

The strain-rate invariant is computed here from the velocities (Cartesian grid), in extended precision, and so
are the laws; every scale is compared, none is skipped.

Tolerance: 1e-12.  The invariant is a sum of squares of some ten roundings each (differences of
neighbouring values are exact to half a unit), 1e-14 in all.  The mean by logarithms, exp of values y up to
745, loses |y| 2^-53 in each of two logarithms and in their sum: 3 * 745 * 1.1e-16 = 2.5e-13.
"""
import numpy as np
import pytest

import sphericalstokes_gb300 as S

pytestmark = pytest.mark.gpu

X = np.longdouble
N = (7, 6, 9)
VSCALES = (0.0, 1e-140, 1e-60, 1e-9, 1.0, 1e9, 1e60, 1e140)
# scales of the old viscosity and of the prefactor
PAIRS = ((1.0, 1.0), (1e-160, 1e160), (1e160, 1e-160), (1e300, 1e-300), (1e-300, 1e300), (1e290, 1e290), (1e-290, 1e-290), (1e-150, 1.0))


def clamped(a):
    """interior cells, with the boundary cells as copies of the nearest interior one"""
    return np.pad(a, 1, mode="edge")


def invariant(p, V):
    """edot_II = sqrt(1/2 sum D_ii^2 + 1/4 (a^2 + b^2 + c^2)) of the clamped interior cells; a, b, c the means of the
    engineering shear rates of a cell's four edges"""
    V1, V2, V3 = (v.astype(X) for v in V)
    d1, d2, d3 = (X((n - 1) / l) for n, l in ((p.n1, p.l1), (p.n2, p.l2), (p.n3, p.l3)))
    D11, D22, D33 = np.diff(V1, axis=0) * d1, np.diff(V2, axis=1) * d2, np.diff(V3, axis=2) * d3
    e12 = np.diff(V2[:, 1:-1, 1:-1], axis=0) * d1 + np.diff(V1[1:-1, :, 1:-1], axis=1) * d2
    e13 = np.diff(V3[:, 1:-1, 1:-1], axis=0) * d1 + np.diff(V1[1:-1, 1:-1, :], axis=2) * d3
    e23 = np.diff(V3[1:-1, :, 1:-1], axis=1) * d2 + np.diff(V2[1:-1, 1:-1, :], axis=2) * d3
    mean = lambda e, i, j: sum(e[tuple(slice(1, None) if (ax == i and s) or (ax == j and t) else slice(None, -1) if ax in (i, j)  # noqa: E731
                                       else slice(None) for ax in range(3))] for s in (0, 1) for t in (0, 1)) / X(4)
    a, b, c = mean(e12, 0, 1), mean(e13, 0, 2), mean(e23, 1, 2)
    inner = (slice(1, -1),) * 3
    x = (D11[inner] ** 2 + D22[inner] ** 2 + D33[inner] ** 2) / X(2) + (a ** 2 + b ** 2 + c ** 2) / X(4)
    return clamped(np.sqrt(x))


def check(got, want):
    """equal to 1e-12, but for results so small that doubles are spaced wider"""
    want = np.where(want > X(np.finfo(np.float64).max), X(np.inf), want)
    np.testing.assert_array_equal(np.isinf(got), np.isinf(want))
    ok = ~np.isinf(want)
    assert np.all(np.isfinite(got[ok]))
    err = np.abs(got[ok].astype(X) - want[ok])
    assert np.all(err <= X(1e-12) * want[ok] + X(1e-320)), float((err / np.maximum(want[ok], X(1e-300))).max())


def edot_params(n_exp, relax, edot_bg):
    return S.default_params("cartesian", n1=N[0], n2=N[1], n3=N[2], rheology="edot_power_relax", n_exp=n_exp, relax=relax,
                            edot_bg=edot_bg, incl_linear=0, init="none")


def run_edot(p, V, eta, ini):
    with S.Solver(p) as sv:
        for f, a in (("ETA", eta), ("ETA_INI", ini), ("PHASE", np.zeros(N))):
            sv.set(f, a)
        for f, a in zip(("V1", "V2", "V3"), V):
            sv.set(f, a)
        sv.power_law()
        return sv.get("ETA")


def velocities(rng, scale):
    return [scale * rng.standard_normal(tuple(n + (i == ax) for i, n in enumerate(N))) for ax in range(3)]


@pytest.mark.parametrize("relax", [0.3, 0.5, 1.0])
@pytest.mark.parametrize("n_exp", [1.0, 1.7, 2.0, 3.0, 4.0, 5.0, 6.0])
@pytest.mark.parametrize("edot_bg", [0.25, 1e-15, 1e20, 1e-158, 1e160])
def test_strain_rates_over_the_range(n_exp, relax, edot_bg):
    rng = np.random.default_rng(1)
    p = edot_params(n_exp, relax, edot_bg)
    for scale in VSCALES:
        V = velocities(rng, scale)
        eta, ini = (np.exp(rng.standard_normal(N)) for _ in range(2))
        got = run_edot(p, V, eta, ini)
        ratio = invariant(p, V) / X(edot_bg)
        t = X(2) * ini.astype(X) / (X(1) + ratio ** ((X(n_exp) - 1) / X(n_exp)))
        check(got, eta.astype(X) ** (X(1) - X(relax)) * t ** X(relax))


@pytest.mark.parametrize("relax", [0.3, 0.5, 0.9])
@pytest.mark.parametrize("n_exp", [1.7, 3.0])
@pytest.mark.parametrize("pair", PAIRS)
def test_old_and_target_viscosity_far_apart(n_exp, relax, pair):
    rng = np.random.default_rng(2)
    p = edot_params(n_exp, relax, 0.25)
    V = velocities(rng, 1.0)
    eta, ini = (s * np.exp(rng.standard_normal(N)) for s in pair)
    eta[2:4, 1, :] = 0.0  # cells without viscosity keep none
    got = run_edot(p, V, eta, ini)
    t = X(2) * ini.astype(X) / (X(1) + (invariant(p, V) / X(0.25)) ** ((X(n_exp) - 1) / X(n_exp)))
    check(got, eta.astype(X) ** (X(1) - X(relax)) * t ** X(relax))
    assert np.all(got[2:4, 1, :] == 0.0)


@pytest.mark.parametrize("n_exp", [1.5, 2.0, 2.5, 3.0])
@pytest.mark.parametrize("scale,tau_C", [(0.0, 1.3), (1e-130, 1e30), (1e-130, 1.0), (1.0, 1.3), (1e130, 1.3), (1e130, 1e-30),
                                         (0.0, 1e-170), (0.0, 1e170), (1e-130, 1e-170), (1e-140, 1e-160), (1e140, 1e160), (1e150, 1e156)])
def test_stresses_over_the_range(n_exp, scale, tau_C):
    rng = np.random.default_rng(3)
    p = S.default_params("spherical", n1=N[0], n2=N[1], n3=N[2], rheology="tau_power", n_exp=n_exp, tau_C=tau_C, init="none")
    with S.Solver(p) as sv:
        for f in ("TAU11", "TAU22", "TAU33", "TAU12", "TAU13", "TAU23"):
            sv.set(f, scale * rng.standard_normal(sv.dims(f)))
        ini = np.exp(rng.standard_normal(N))
        for f in ("ETA", "ETA_INI"):
            sv.set(f, ini)
        sv.set("PHASE", np.zeros(N))
        sv.power_law()
        tii, got = sv.get("TII"), sv.get("ETA")
    power = (tii.astype(X) / X(tau_C)) ** (X(n_exp) - 1)
    # (power_law! takes 1/eta_PL: infinite, and eta zero, where eta_PL = eta_ini / power is below 1 / the largest double)
    gone = power / ini > X(np.finfo(np.float64).max)
    check(got, np.where(gone, X(0), X(2) * ini.astype(X) / (X(1) + power)))


@pytest.mark.parametrize("n_exp", [2.0, 2.5, 3.0, 5.0])
@pytest.mark.parametrize("scale,tau_C", [(1.0, 1.3), (1e-130, 1e-160), (1e140, 1e158), (1e150, 1e156)])
def test_relaxed_stresses_over_the_range(n_exp, scale, tau_C):
    rng = np.random.default_rng(4)
    relax = 0.3
    p = S.default_params("cylindrical", n1=N[0], n2=N[1], n3=N[2], rheology="tau_power_relax", n_exp=n_exp, relax=relax, tau_C=tau_C, init="none")
    with S.Solver(p) as sv:
        for f in ("TAU11", "TAU22", "TAU33", "TAU12", "TAU13", "TAU23"):
            sv.set(f, scale * rng.standard_normal(sv.dims(f)))
        ini, old = (np.exp(rng.standard_normal(N)) for _ in range(2))
        for f, a in (("ETA", ini), ("ETA_INI", ini), ("ETA_PL", old), ("PHASE", np.zeros(N))):
            sv.set(f, a)
        sv.power_law()
        tii, got, pl = sv.get("TII"), sv.get("ETA"), sv.get("ETA_PL")
    want = (ini.astype(X) * (tii.astype(X) / X(tau_C)) ** (X(1) - X(n_exp))) ** X(relax) * old.astype(X) ** (X(1) - X(relax))
    check(pl, want)
    check(got, X(2) / (X(1) / ini.astype(X) + X(1) / want))
