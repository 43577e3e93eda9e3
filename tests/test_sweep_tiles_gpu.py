"""The fused sweep at the edges of its tiling: 32 x 14 tiles, chunks of 1 plane up to the whole
grid, the smallest grid, for the correction problem (k_sweep<G, 1>, which also writes the ghost
velocities or evaluates them where it reads them) against the FP64 oracle, and for the FP32
reference iteration (k_sweep<G, 0>) against the FP32 kernels of one reference step each.

Tolerances: the FP32 bound of test_sweep_parity_gpu (2e-4 of a group's max-norm) against FP64: a
handful of sweeps accumulate well under 100 roundings of 6e-8 per value, amplified by the
differences of neighbouring stresses.  Between two FP32 evaluations of the same expressions from
the same FP32 state, 1e-5 (the rounding of the FP32 state itself, which the scripts' r = 1000
geometry amplifies, is common to both).
"""
import numpy as np
import pytest

import sphericalstokes_gb300 as S
from test_sweep_parity_gpu import TOL, case_params, run_case

pytestmark = pytest.mark.gpu

SIZES = [(5, 5, 5), (31, 13, 6), (32, 14, 7), (33, 15, 9), (30, 28, 5), (65, 29, 11)]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("geometry,bc", [("spherical", "stress"), ("spherical", "free_surface"), ("spherical", "free_slip"),
                                         ("cylindrical", "diapir"), ("cartesian", "diapir")])
@pytest.mark.parametrize("chunk", [1, 2, 5, 99])
def test_correction_sweep_tile_edges(monkeypatch, geometry, bc, n, chunk):
    monkeypatch.setenv("SPH_FUSED_CHUNK", str(chunk))
    p = case_params(geometry, n, bc)
    if bc == "free_surface":
        S.set_params(p, rheology="linear", fs_kappa=0.1)
    err = run_case(p, 5, random_start=True, seed=chunk)
    assert max(err.values()) < TOL, err


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("geometry", ["spherical", "cylindrical", "cartesian"])
def test_fp32_iteration_tile_edges(monkeypatch, geometry, n):
    monkeypatch.setenv("SPH_FUSED_CHUNK", "2")
    p = S.default_params(geometry, n1=n[0], n2=n[1], n3=n[2], rheology="linear", precision="fp32", n_exp=1.0, vr=10.0)
    got = []
    for kernels in ("auto", "simple"):
        S.set_params(p, kernels=kernels)
        with S.Solver(p) as sv:
            sv.step(5)
            got.append({f: sv.get(f) for f in ("P", "V1", "V2", "V3")})
    scale = {"P": np.abs(got[1]["P"]).max(), "V": max(np.abs(got[1][f]).max() for f in ("V1", "V2", "V3"))}
    for f, a in got[0].items():
        assert np.abs(a - got[1][f]).max() < 1e-5 * scale[f[0]], f
