"""The FP64 viscosity laws over the range of their arguments: the table-driven power, quotient and
root of sph_math.cuh against numpy's pow / exp / log, with arguments from zero through the whole
double range (outside its normal numbers the kernels take CUDA's functions).

Tolerance: numpy's own evaluation (log, exp of values up to a few hundred) is good to some 100
units in the last place at the ends of the range, 1e-13; the kernels' power is good to about one.
"""
import numpy as np
import pytest

import sphericalstokes_gb300 as S

pytestmark = pytest.mark.gpu

RTOL = 1e-13
SCALES = (0.0, 1e-150, 1e-20, 1e-3, 1.0, 7.0, 1e4, 1e30, 1e140)
TAUS = ("TAU11", "TAU22", "TAU33", "TAU12", "TAU13", "TAU23")


@pytest.mark.parametrize("geometry", ["spherical", "cylindrical", "cartesian"])
@pytest.mark.parametrize("n_exp,relax", [(1.5, 1e-3), (3.0, 0.5), (5.0, 1.0), (1.0, 0.3)])
@pytest.mark.parametrize("n", [(5, 6, 7), (33, 9, 5)])
def test_stress_power_law(geometry, n_exp, relax, n):
    law = "tau_power" if geometry == "spherical" else "tau_power_relax"
    p = S.default_params(geometry, n1=n[0], n2=n[1], n3=n[2], rheology=law, n_exp=n_exp, relax=relax, tau_C=1.3)
    rng = np.random.default_rng(0)
    with S.Solver(p) as sv:
        for scale in SCALES:
            for f in TAUS:
                sv.set(f, scale * rng.standard_normal(sv.dims(f)))
            ini, old = np.exp(3 * rng.standard_normal(sv.dims("ETA"))), np.exp(3 * rng.standard_normal(sv.dims("ETA")))
            sv.set("ETA_INI", ini)
            sv.set("ETA_PL", old)
            sv.set("ETA", ini)
            sv.power_law()
            tii, eta, pl = sv.get("TII"), sv.get("ETA"), sv.get("ETA_PL")
            if law == "tau_power_relax" and n_exp <= 1.0:
                np.testing.assert_array_equal(eta, ini)
                continue
            with np.errstate(divide="ignore", over="ignore", invalid="ignore"):
                want = ini * (tii / p.tau_C) ** (1.0 - n_exp)
                if law == "tau_power_relax":
                    want = np.exp(np.log(want) * relax + np.log(old) * (1.0 - relax))
                    np.testing.assert_allclose(pl, want, rtol=RTOL)
                np.testing.assert_allclose(eta, 2.0 / (1.0 / ini + 1.0 / want), rtol=RTOL)


@pytest.mark.parametrize("n_exp,relax", [(1.0, 0.5), (1.7, 0.5), (3.0, 0.3), (5.0, 1.0)])
@pytest.mark.parametrize("n", [(5, 6, 7), (33, 9, 5)])
def test_strain_rate_power_law(n_exp, relax, n):
    """A velocity field V = (a r) e_r has the strain rates of a uniform expansion: D_ii = a - div/3 = 0 up
    to rounding, so a shear V_φ = a r sinθ (θ - π/2) is added: the invariant comes from the kernel itself at
    n = 1e9 (η_t with exponent -1 is η_ini ε̇_bg / ε̇ in the limit), other exponents are compared with it."""
    p = S.sector_params(n, bc="free_slip", rheology="edot_power_relax", n_exp=1e9, relax=1.0, edot_bg=0.7, incl_linear=0, vr=1.0)
    rng = np.random.default_rng(1)
    with S.Solver(p) as sv:
        for scale in SCALES[1:]:
            V = {f: scale * rng.standard_normal(sv.dims(f)) for f in ("V1", "V2", "V3")}
            for f, a in V.items():
                sv.set(f, a)
            one = np.ones(sv.dims("ETA"))
            S.set_params(p, n_exp=1e9, relax=1.0)
            sv.update_params(p)
            sv.set("ETA_INI", one)
            sv.set("ETA", one)
            sv.power_law()
            q = 2.0 / sv.get("ETA") - 1.0  # (ε̇/ε̇_bg)^(1 - 1e-9)
            if not (q.min() > 1e-2 and q.max() < 1e8):
                continue  # the invariant cannot be read back from η to full accuracy
            ini, old = np.exp(3 * rng.standard_normal(one.shape)), np.exp(3 * rng.standard_normal(one.shape))
            S.set_params(p, n_exp=n_exp, relax=relax)
            sv.update_params(p)
            sv.set("ETA_INI", ini)
            sv.set("ETA", old)
            sv.power_law()
            ratio = q ** (1.0 / (1.0 - 1e-9))
            et = 2.0 * ini / (1.0 + ratio ** ((n_exp - 1.0) / n_exp))
            # reading ε̇ back from η loses up to (1 + 1/q) roundings
            np.testing.assert_allclose(sv.get("ETA"), np.exp((1.0 - relax) * np.log(old) + relax * np.log(et)), rtol=1e-12)
