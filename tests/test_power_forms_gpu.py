"""Exponents around the edges of the forms that replace the table-driven power: products for integer n up
to 13 in the stress law (odd and even powers, the largest, the first beyond), roots for n = 2 .. 5 in the
strain-rate law (each p/q, the first beyond).  Same comparison and tolerance as for other exponents."""
import pytest

import test_fp64_laws_gpu as laws

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geometry", ["spherical", "cartesian"])
@pytest.mark.parametrize("n_exp", [2.0, 4.0, 8.0, 13.0, 14.0])
@pytest.mark.parametrize("n", [(5, 5, 5), (33, 6, 7)])
def test_stress_law_products(geometry, n_exp, n):
    laws.test_stress_power_law(geometry, n_exp, 0.3, n)


@pytest.mark.parametrize("n_exp", [2.0, 4.0, 6.0])
@pytest.mark.parametrize("n", [(5, 5, 5), (33, 6, 7)])
def test_strain_rate_law_roots(n_exp, n):
    laws.test_strain_rate_power_law(n_exp, 0.4, n)
