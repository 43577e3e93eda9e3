"""The boundary program as launched (faces, edges and corners in one or two launches) against the
oracle's stage-by-stage kernels, on every boundary set and geometry, at grid sizes around the warp
width and at the smallest grid.  Every entry of the velocities starts random, ghosts included.

Tolerance: copies are exact; a divergence-free ghost is some ten FP64 operations and a quotient
of values near 1 in magnitude, 1e-12 of the field's largest entry.  The cylindrical and Cartesian
oracle has no boundary kernels of its own: their stages are written out here
(CylindricalStokes_diapir.jl:358-366, CartesianStokes_diapir.jl:371-379)."""
import numpy as np
import pytest

import oracle
import sphericalstokes_gb300 as S
from sphericalstokes_gb300.plateau import linspace
from test_parity_gpu import compare, randomize, relerr

pytestmark = pytest.mark.gpu

SIZES = [(5, 5, 5), (5, 34, 33), (33, 5, 66), (35, 32, 5), (131, 7, 31)]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("bc", ["diapir", "free_slip", "stress", "free_surface"])
def test_spherical_ghosts(bc, n):
    if bc in ("diapir", "free_slip"):
        p = S.default_params("spherical", n1=n[0], n2=n[1], n3=n[2], bc=bc)
    else:
        p = S.sector_params(n, bc=bc, rheology="linear", sig_bc=(0.0, 0.5, -0.5))
    with S.Solver(p) as sv:
        o = oracle.Sph.from_params(p)
        randomize(o, sv, np.random.default_rng(11), ("V1", "V2", "V3"))
        sv.apply_bc()
        o.apply_bc()
        compare(o, sv, ["V1", "V2", "V3"], 1e-12)


STAGES = {  # per axis: what each of V1, V2, V3 does on both faces
    "cylindrical": [("neg", "copy", "copy"), ("zero", "neg", "lin"), ("zero", "zero", "lin2m")],
    "cartesian": [("lin2m", "zero", "zero"), ("lin", "neg", "zero"), ("copy", "copy", "neg")],
}


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("geometry", ["cylindrical", "cartesian"])
def test_diapir_ghosts(geometry, n):
    p = S.default_params(geometry, n1=n[0], n2=n[1], n3=n[2])
    x2 = linspace(p.c2, p.l2, p.n2) * (p.sh * (p.r if geometry == "cylindrical" else 1.0))
    rng = np.random.default_rng(11)
    with S.Solver(p) as sv:
        V = [rng.standard_normal(sv.dims(f)) for f in ("V1", "V2", "V3")]
        for f, a in zip(("V1", "V2", "V3"), V):
            sv.set(f, a)
        sv.apply_bc()
        for ax, ops in enumerate(STAGES[geometry]):
            for a, kind in zip(V, ops):
                for b, inner in ((0, 1), (-1, -2)):
                    ghost, src = np.moveaxis(a, ax, 0)[b], np.moveaxis(a, ax, 0)[inner]
                    lin = x2[b] if ax == 1 else x2[:, None] if ax == 0 else x2[None, :]
                    if kind.startswith("lin"):
                        ghost[...] = lin if kind == "lin" else 2.0 * lin - src
                    else:
                        ghost[...] = {"neg": -1.0, "copy": 1.0, "zero": 0.0}[kind] * src
        for f, a in zip(("V1", "V2", "V3"), V):
            assert relerr(sv.get(f), a) < 1e-12, f
