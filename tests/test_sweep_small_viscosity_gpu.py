"""FP32 sweeps where viscosities are so small that the divisors of the stress update and of the pseudo-step are subnormal
numbers, against the cp.async sweep (another kernel, quotients by CUDA's __fdividef).

Tolerance: a subnormal number of 1e-40 has 16 bits; each quotient and product of two such numbers is good to 2^-15, a sweep
chains four (ratio, stress, stress difference, pseudo-step), and differences of neighbours lose as much again:
8 * 2^-15 = 2.5e-4 of the field's largest value, times the sweeps.
"""
import numpy as np
import pytest

import sphericalstokes_gb300 as S

pytestmark = pytest.mark.gpu

TOL = 2.5e-4
STATE = ("dP", "dV1", "dV2", "dV3", "dTAU11", "dTAU22", "dTAU33", "dTAU12", "dTAU13", "dTAU23")
GEOM = {"spherical": lambda n, q: S.sector_params(n, bc="stress", rheology="linear", precision=q),
        "cylindrical": lambda n, q: S.default_params("cylindrical", n1=n[0], n2=n[1], n3=n[2], rheology="linear", bc="stress", precision=q),
        "cartesian": lambda n, q: S.default_params("cartesian", n1=n[0], n2=n[1], n3=n[2], rheology="linear", precision=q)}


def viscosity(n, kind, rng):
    eta = 1e-39 * (1.0 + rng.random(n))
    if kind == "block":  # a block of it in ordinary viscosity
        out = np.ones(n)
        out[2:7, 1:6, 2:8] = eta[2:7, 1:6, 2:8]
        return out
    return eta


def run(p, kind, sweeps, by_caller=False):
    rng = np.random.default_rng(1)
    n = (p.n1, p.n2, p.n3)
    eta = viscosity(n, kind, rng)
    with S.Solver(p) as sv:
        zero = np.zeros(n)
        sv.set("RHO", zero)
        for f in ("P", "V1", "V2", "V3"):
            sv.set(f, np.zeros(sv.dims(f)))
        V = {f: (1e2 if kind == "everywhere" else 1e-3) * rng.standard_normal(sv.dims(f)) for f in ("V1", "V2", "V3")}
        if p.precision == S.PREC["fp32"]:
            sv.set("ETA", eta)
            for f, a in V.items():
                sv.set(f, a)
            sv.step(sweeps)
            return {f: sv.get(f) for f in ("P", "V1", "V2", "V3", "TAU11", "TAU22", "TAU33", "TAU12", "TAU13", "TAU23")}
        if not by_caller:
            sv.set("ETA", eta)
        sv.corr_get("dP")  # (the correction problem is prepared)
        if by_caller:
            sv.corr_set("ETA", eta)
            sv.corr_set("ETA_SM", eta)
        for f, a in V.items():
            sv.corr_set("d" + f, a)
        sv.sweep(sweeps)
        return {f: sv.corr_get(f) for f in STATE}


def compare(monkeypatch, make, kind, sweeps, by_caller=False):
    got = run(make(), kind, sweeps, by_caller)
    monkeypatch.setenv("SPH_NO_TMA", "1")
    want = run(make(), kind, sweeps, by_caller)
    for f in want:
        scale = np.abs(want[f]).max()
        assert np.all(np.isfinite(want[f])) and scale > 0.0, f
        assert np.all(np.isfinite(got[f])), f
        assert np.abs(got[f] - want[f]).max() <= TOL * sweeps * scale, (f, np.abs(got[f] - want[f]).max() / scale)


@pytest.mark.parametrize("geometry", GEOM)
@pytest.mark.parametrize("kind,sweeps", [("everywhere", 3), ("block", 1)])
@pytest.mark.parametrize("n", [(13, 11, 9), (35, 16, 10)])
def test_correction_sweeps(monkeypatch, geometry, kind, sweeps, n):
    compare(monkeypatch, lambda: GEOM[geometry](n, "mixed"), kind, sweeps)


@pytest.mark.parametrize("geometry", GEOM)
def test_iterations(monkeypatch, geometry):
    compare(monkeypatch, lambda: GEOM[geometry]((13, 11, 9), "fp32"), "everywhere", 2)


def test_viscosity_set_by_the_caller(monkeypatch):
    compare(monkeypatch, lambda: GEOM["spherical"]((13, 11, 9), "mixed"), "everywhere", 2, by_caller=True)


def test_ordinary_sweeps_are_the_same_on_both_paths():
    """a state of ordinary viscosity on the path for small ones: the same bits"""
    out = []
    for by_caller in (False, True):
        with S.Solver(GEOM["spherical"]((33, 15, 12), "mixed")) as sv:
            if by_caller:
                sv.corr_set("ETA", sv.corr_get("ETA"))
            rng = np.random.default_rng(2)
            for f in ("dV1", "dV2", "dV3"):
                sv.corr_set(f, 1e-3 * rng.standard_normal(sv.corr_get(f).shape))
            sv.sweep(4)
            out.append({f: sv.corr_get(f) for f in STATE})
    for f in STATE:
        np.testing.assert_array_equal(out[0][f], out[1][f])


def test_batch_with_one_small_viscosity():
    """solves of a batch with ordinary and with small viscosities: the same bits as alone"""
    def solvers():
        out = []
        for i, geometry in enumerate(GEOM):
            sv = S.Solver(GEOM[geometry]((13 + i, 11, 9), "mixed"))
            n = (13 + i, 11, 9)
            if i == 1:
                sv.set("RHO", np.zeros(n))
                sv.set("ETA", viscosity(n, "block", np.random.default_rng(4)))
            out.append(sv)
        return out
    kw = dict(tol=1e-30, maxiter=40, nout=10, criterion="residual", max_outer=2, inner_max=20)
    alone, together = solvers(), solvers()
    try:
        for sv in alone:
            sv.solve(**kw)
        S.solve_batch(together, S.make_opts(**kw))
        for a, b in zip(alone, together):
            for f in ("P", "V1", "V2", "V3"):
                np.testing.assert_array_equal(a.get(f), b.get(f))
    finally:
        for sv in alone + together:
            sv.close()
