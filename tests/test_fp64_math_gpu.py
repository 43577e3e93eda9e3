"""The FP64 primitives of sph_math.cuh, element by element: quotients and roots against the IEEE operations,
powers against extended precision.

Tolerances, from the approximate reciprocal and reciprocal root (relative error e of about 2^-20, at most 2^-19):
quotient and root carry e^4 = 2^-76 before their last rounding, so a result differs from the correctly
rounded one where the exact value lies that close to a midpoint, one pair in 2^22; never by more than one
unit.  Of 2^20 pairs at most four may differ.  Table-driven power: 1.1 units in the last place as its
comment derives, 1.1 * 2^-52 at most in relative terms.  Root of a power: Halley's step cubes an error of 1e-6
to 1e-18, two roundings of the correction and one of the sum: one unit.
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from sphericalstokes_gb300 import build

pytestmark = pytest.mark.gpu

X = np.longdouble
M = 1 << 20
ULP = 2.0 ** -52


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = tmp_path_factory.mktemp("probe") / "libprobe.so"
    src = Path(__file__).with_name("fp64_math_probe.cu")
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, f"-I{build.CSRC}", "-o", str(so), str(src)], check=True, capture_output=True)
    lib = C.CDLL(str(so))
    pd = C.POINTER(C.c_double)
    lib.probe.argtypes = [C.c_int, C.c_longlong, pd, pd, pd, C.c_int, C.c_int, C.c_double]

    def run(op, a, b=None, p=1, q=3, c=0.0):
        a = np.ascontiguousarray(a, dtype=np.float64)
        b = np.ascontiguousarray(a if b is None else b, dtype=np.float64)
        out = np.empty_like(a)
        rc = lib.probe(op, a.size, *(x.ctypes.data_as(pd) for x in (a, b, out)), p, q, c)
        assert rc == 0, rc
        return out
    return run


def numbers(rng, lo, hi, n=M):
    """random mantissas, exponents spread evenly over 2^lo .. 2^hi"""
    return np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))


def nearly_ieee(got, want, allowed):
    bad = got != want
    assert np.count_nonzero(bad) <= allowed, np.count_nonzero(bad)
    assert np.all(np.abs(got[bad] - want[bad]) <= np.spacing(np.abs(want[bad])))


@pytest.mark.parametrize("lo,hi", [(-1, 1), (-30, 30), (-400, 400)])
def test_near_div_is_the_ieee_quotient(probe, lo, hi):
    rng = np.random.default_rng(1)
    a, b = numbers(rng, lo, hi), numbers(rng, lo, hi)
    nearly_ieee(probe(0, a, b), a / b, 4)
    nearly_ieee(probe(0, a, a + b), a / (a + b), 4)


@pytest.mark.parametrize("ea", [-1022, -501, -499, 0, 498, 500, 1022])
@pytest.mark.parametrize("eb", [-1022, -501, -499, 0, 498, 500, 1022])
def test_near_div_over_the_range(probe, ea, eb):
    """the edges of the range whose quotients are formed without the IEEE division, overflow and underflow"""
    rng = np.random.default_rng(5)
    a, b = numbers(rng, ea, ea + 2, 1 << 12), numbers(rng, eb, eb + 2, 1 << 12)
    with np.errstate(over="ignore", under="ignore"):
        nearly_ieee(probe(0, a, b), a / b, 0)


def test_near_div_of_any_operand(probe):
    v = [0.0, 5e-324, 1e-310, 2.3e-308, 1e-200, 1e-155, 1.0, 1e155, 1e200, 1e300, 1.79e308, np.inf, np.nan]
    v = np.array(v + [-x for x in v])
    a, b = (x.ravel() for x in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        np.testing.assert_array_equal(probe(0, a, b), a / b)
        np.testing.assert_array_equal(np.signbit(probe(0, a, b))[~np.isnan(a / b)], np.signbit(a / b)[~np.isnan(a / b)])


@pytest.mark.parametrize("lo,hi", [(-1, 1), (-20, 20), (-60, 60)])
def test_ghost_quotient_is_the_ieee_quotient(probe, lo, hi):
    """FP32: the error of the reciprocal, 2^-23, squared by the residual step: 2^-46 before the last rounding, so that one
    pair in 2^21 may differ"""
    rng = np.random.default_rng(6)
    a, b = numbers(rng, lo, hi).astype(np.float32), numbers(rng, lo, hi).astype(np.float32)
    nearly_ieee(probe(5, a, b).astype(np.float32), a / b, 4)


@pytest.mark.parametrize("lo,hi", [(-1, 1), (-30, 30), (-1000, 1000)])
def test_fast_sqrt_is_the_ieee_root(probe, lo, hi):
    a = numbers(np.random.default_rng(2), lo, hi)
    nearly_ieee(probe(2, a), np.sqrt(a), 4)


def test_fast_sqrt_of_any_operand(probe):
    a = np.array([0.0, -0.0, 5e-324, 1e-310, 2.3e-308, 1e308, 1.79e308, np.inf, np.nan, -1.0])
    with np.errstate(invalid="ignore"):
        np.testing.assert_array_equal(probe(2, a), np.sqrt(a))


@pytest.mark.parametrize("c", [0.0, 0.25, 1.0 / 3.0, 0.5, 0.9, 1.0, -0.25, 1.35, 2.0])
def test_fast_pow(probe, c):
    x = numbers(np.random.default_rng(3), -450, 450, 1 << 16)
    want = x.astype(X) ** X(c)
    assert np.max(np.abs((probe(3, x, c=c).astype(X) - want) / want)) <= 1.1 * ULP


def test_fast_pow_of_any_operand(probe):
    x = np.array([0.0, 5e-324, 1e-310, 2.3e-308, 1e308, np.inf, np.nan, 1.0])
    for c in (0.25, 0.5, -0.5, 0.0):
        with np.errstate(divide="ignore"):
            np.testing.assert_allclose(probe(3, x, c=c), x ** c, rtol=2 * ULP)  # (CUDA's pow: two units)


@pytest.mark.parametrize("p,q", [(1, 4), (1, 3), (3, 8), (2, 5)])
def test_root_pow(probe, p, q):
    x = numbers(np.random.default_rng(4), -295, 295, 1 << 16)
    want = x.astype(X) ** (X(p) / X(q))
    assert np.max(np.abs((probe(4, x, p=p, q=q).astype(X) - want) / want)) <= ULP
