"""Workloads of the solver that its performance is judged on, through the package's public entry points.

Kinds of pass (``case["kind"]``):

``pt``       the state of a checkpoint up, k reference PT iterations (``Solver.step``) or the script's whole
             loop with its exit check (``Solver.solve`` on the reference criterion), in FP64 or FP32, fields back.
``mixed``    one defect-correction step of the mixed-precision solve: the step's fields up, k FP32
             sweeps inside the FP64 residual (``Solver.solve`` with an iteration budget), fields back.
``batch``    the same for several uneven grids at once (``solve_batch``).
``adjoint``  k iterations of the transposed solve and the parameter gradients (``adjoint.adjoint_solve``,
             ``adjoint.vjp``, ``adjoint.law_vjp``).

Velocities and pressures that come out of FP32 arithmetic are handed on as float32.

``exact`` iterates the same discrete equations in 64 bits with torch (:class:`Model`).
"""
import math

import numpy as np
import torch

import sphericalstokes_gb300 as S
from sphericalstokes_gb300 import adjoint, batch, plateau

VEL = ("V1", "V2", "V3")
TAU = ("TAU11", "TAU22", "TAU33", "TAU12", "TAU13", "TAU23")


# ---------------------------------------------------------------------------
# cases
def listed():
    return [
        # the plateau script on its own 70 x 5 x 5 grid: one continuation step, a check every 10 iterations
        dict(name="plateau_70x5x5_fp64", kind="pt", setup="plateau", precision="fp64", n1=70, n2=5, n3=5, k=200, n_exp=1.0),
        # the spherical diapir script (stress power law) at the size of a first run
        dict(name="diapir_sph_63_fp64", kind="pt", setup="spherical", precision="fp64", n1=63, n2=63, n3=63, k=40, n_exp=3.0),
        # the Cartesian script at its default 207 cells a side
        dict(name="diapir_cart_207_fp64", kind="pt", setup="cartesian", precision="fp64", n1=207, n2=207, n3=207, k=10, n_exp=5.0),
        # plain FP64 iterations of the strain-rate-law sector under far-field stress (the comparison every mixed solve is held to)
        dict(name="sector_127_fp64", kind="pt", setup="sector", precision="fp64", n1=127, n2=127, n3=127, k=20, n_exp=3.0),
        # FP32 iterations of the cylindrical script, ragged grid
        dict(name="diapir_cyl_95x79x67_fp32", kind="pt", setup="cylindrical", precision="fp32", n1=95, n2=79, n3=67, k=200, n_exp=3.0),
        # a small linear solve of a parameter study
        dict(name="mixed_cart_47x31x39", kind="mixed", setup="cartesian", n1=47, n2=31, n3=39, k=1000, n_exp=1.0),
        # the 63^3 sector of the time-to-tolerance runs
        dict(name="mixed_sector_63", kind="mixed", setup="sector", n1=63, n2=63, n3=63, k=1000, n_exp=3.0),
        # an odd grid between the benchmark's sizes
        dict(name="mixed_sector_131x117x101", kind="mixed", setup="sector", n1=131, n2=117, n3=101, k=1000, n_exp=3.0),
        # the headline 255^3 sector
        dict(name="mixed_sector_255", kind="mixed", setup="sector", n1=255, n2=255, n3=255, k=500, n_exp=3.0),
        # the elliptical plateau with its free-surface top: the largest grid of the configurations
        dict(name="mixed_plateau_511x255x255", kind="mixed", setup="ellipse", n1=511, n2=255, n3=255, k=300, n_exp=3.0),
        # a lockstep batch of uneven grids in all three geometries
        dict(name="batch_12", kind="batch", count=12, draw_seed=3, edge_lo=31, edge_hi=47, k=600),
        # the transposed solve and the gradients of a surface misfit
        dict(name="adjoint_sector_63", kind="adjoint", setup="sector", n1=63, n2=63, n3=63, k=60, n_exp=3.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("pt", "pt", "mixed", "mixed", "mixed", "batch", "adjoint"))
    if kind == "batch":
        lo = rng.choice((31, 47))
        return dict(kind="batch", count=rng.randint(4, 16), draw_seed=rng.randint(0, 999), edge_lo=lo, edge_hi=lo + 16, k=200 * rng.randint(1, 3))
    if kind == "pt":
        setup = rng.choice(("spherical", "cylindrical", "cartesian", "sector"))
        n = [_log_int(rng, 15, 191) for _ in range(3)]
        cells = n[0] * n[1] * n[2]
        precision = rng.choice(("fp64", "fp32"))
        k = max(4, min(200, int((2e7 if precision == "fp64" else 4e8) / cells)))
        return dict(kind="pt", setup=setup, precision=precision, n1=n[0], n2=n[1], n3=n[2], k=2 * (k // 2),
                    n_exp=rng.choice((2.0, 3.0) if setup == "spherical" else (2.0, 3.0, 4.0, 5.0)))  # unrelaxed above 3: unstable
    if kind == "mixed":
        setup = rng.choice(("sector", "sector", "cylindrical", "cartesian", "ellipse"))
        n = [_log_int(rng, 23, 255) for _ in range(3)]
        k = max(100, min(1000, int(5e9 / (n[0] * n[1] * n[2]))))
        return dict(kind="mixed", setup=setup, n1=n[0], n2=n[1], n3=n[2], k=100 * (k // 100), n_exp=rng.choice((1.0, 2.0, 3.0)))
    n = [_log_int(rng, 11, 95) for _ in range(3)]
    k = max(4, min(100, int(1.5e7 / (n[0] * n[1] * n[2]))))
    return dict(kind="adjoint", setup="sector", n1=n[0], n2=n[1], n3=n[2], k=k, n_exp=rng.choice((1.0, 3.0)))


# ---------------------------------------------------------------------------
# inputs
def params(case):
    """The solver parameters of a case on one grid."""
    n = (case["n1"], case["n2"], case["n3"])
    precision = case.get("precision", {"mixed": "mixed"}.get(case["kind"], "fp64"))
    script = case["kind"] == "pt" and case["setup"] != "sector"  # the scripts' own stress power law, in the inclusion too
    kw = dict(n1=n[0], n2=n[1], n3=n[2], precision=precision, init="none", incl_linear=0 if script else 1)
    if case["setup"] == "plateau":
        p = plateau.PlateauSetup(nr=n[0], nth=n[1], nph=n[2]).params(precision, n_exp=case["n_exp"])
        p.vpdt = p.l1 / (p.n1 - 1) / (2.0 + 4.5 * math.log10(p.vr))
        return p
    if case["setup"] == "ellipse":
        setup = plateau.EllipsePlateau(nr=n[0], nth=n[1], nph=n[2], top="free_surface", n_exp=case["n_exp"])
        p = setup.params(precision)
        p.vpdt = 0.25 * p.l1 / (p.n1 - 1) / (2.0 + 4.5 * math.log10(p.vr))  # the stable quarter of the script's step
        return p
    law = dict(rheology="linear") if case["n_exp"] == 1.0 else dict(rheology="edot_power_relax", n_exp=case["n_exp"], relax=0.5, edot_bg=0.25)
    if case["setup"] == "sector":
        p = S.sector_params(n, vr=1e2, bc="stress", sig_bc=(0.0, 0.5, -0.5), **law)
    else:
        if script:
            power = "tau_power" if case["setup"] == "spherical" else "tau_power_relax"
            law = dict(rheology=power, n_exp=case["n_exp"], switch_err=0.0)
        p = S.default_params(case["setup"], vr=1e2, rho_in=-1.0, **law)
    S.set_params(p, **kw)
    if p.vpdt <= 0.0:  # the scripts' step, from the smallest spacing of the grid
        h = min(p.l1 / (p.n1 - 1), 6.0 / (p.n2 - 1), 6.0 / (p.n3 - 1))
        p.vpdt = h / (2.0 + 4.5 * math.log10(p.vr))
    p.vpdt *= 0.5  # stable on ragged grids too
    return p


def _axes(p, dev):
    def line(c, l, n):
        lo, hi = c - l / 2.0, c + l / 2.0
        x = lo + (hi - lo) * torch.arange(n, dtype=torch.float64, device=dev) / (n - 1)
        x[-1] = hi
        return x
    return line(p.c1, p.l1, p.n1), line(p.c2, p.l2, p.n2), line(p.c3, p.l3, p.n3)


def _extent(p, f):
    n = [p.n1, p.n2, p.n3]
    if f in VEL:
        n[VEL.index(f)] += 1
    return n


def fields(p, seed, dev="cuda"):
    """Density, viscosity, linear-cell flag, top load and a smooth flow, on the grid of ``p``: an inclusion
    at a seeded place (a crust over a mantle for the plateaus), seeded noise on both, low modes in V."""
    g = torch.Generator(device=dev).manual_seed(int(seed))
    x1, x2, x3 = _axes(p, dev)
    unit = [((x - x[0]) / (x[-1] - x[0])) for x in (x1, x2, x3)]
    u1, u2, u3 = unit[0].view(-1, 1, 1), unit[1].view(1, -1, 1), unit[2].view(1, 1, -1)
    r = torch.rand(32, generator=g, device=dev, dtype=torch.float64).tolist()
    shape = (p.n1, p.n2, p.n3)
    top_down = p.bc == S.BC["free_surface"] or (p.bc == S.BC["free_slip"] and p.rheology == S.RHEO["tau_power"])
    if top_down:  # a crust whose thickness follows an elliptical plateau
        e2 = ((u2 - 0.5) / 0.3) ** 2 + ((u3 - 0.5) / 0.15) ** 2
        w = torch.exp(-e2 * (0.8 + 0.4 * r[0]))
        inside = ((1.0 - u1) < 0.175 * (1.0 + w)).expand(shape)
        rho_in, rho_out, e_in, e_out = 2800.0 / 3300.0, 1.0, 1e-2, 1.0
    else:
        d2 = (u1 - 0.4 - 0.2 * r[0]) ** 2 + (u2 - 0.4 - 0.2 * r[1]) ** 2 + (u3 - 0.4 - 0.2 * r[2]) ** 2
        inside = (d2 < 0.03).expand(shape)
        rho_in, rho_out, e_in, e_out = p.rho_in, p.rho0, 1.0 / p.vr, 1.0
    noise = lambda: torch.randn(shape, generator=g, device=dev, dtype=torch.float64)  # noqa: E731
    one = torch.ones(shape, dtype=torch.float64, device=dev)
    rho = torch.where(inside, rho_in * one, rho_out * one) * (1.0 + 0.02 * noise()) + 0.02 * noise()
    eta = torch.where(inside, e_in * one, e_out * one) * torch.exp(0.1 * noise())
    f = {"RHO": rho, "ETA": eta, "ETA_INI": eta.clone()}
    linear = inside if not top_down else ~inside
    f["PHASE"] = linear.to(torch.float64) if p.incl_linear else torch.zeros_like(eta)
    if p.rheology == S.RHEO["tau_power_relax"]:
        f["ETA_PL"] = eta.clone()
    if p.bc == S.BC["free_surface"]:
        f["TOP_LOAD"] = torch.zeros_like(eta)
        f["TOP_LOAD"][-1] = 0.03 * w[0]
    for m, name in enumerate(VEL):
        u = [torch.linspace(0, 1, n, dtype=torch.float64, device=dev) for n in _extent(p, name)]
        q = r[4 + 8 * m:12 + 8 * m]
        a = [torch.sin(math.pi * ((1 + i) * u[i] + q[i])) + 0.3 * torch.cos(2 * math.pi * (u[i] + q[3 + i])) for i in range(3)]
        amp = (0.05 if p.bc != S.BC["free_surface"] else 0.005) * p.g
        f[name] = amp * (0.5 + q[6]) * a[0].view(-1, 1, 1) * a[1].view(1, -1, 1) * a[2].view(1, 1, -1)
    f["P"] = 0.01 * p.g * torch.sin(math.pi * (u1 + u2 + r[3])) * torch.cos(math.pi * u3)
    return f


def _host(t):
    """A field in page-locked memory, in the layout that the solver takes (first axis fastest)."""
    h = torch.empty(t.numel(), dtype=torch.float64, pin_memory=True)
    h.view(tuple(reversed(t.shape))).copy_(t.permute(2, 1, 0))
    return h.numpy().reshape(tuple(t.shape), order="F")


def _buffers(p, names):
    """Page-locked arrays that a program reads fields into, and float32 ones for FP32 results."""
    out = {}
    for f in names:
        n = _extent(p, f)
        h = torch.empty(n[0] * n[1] * n[2], dtype=torch.float64, pin_memory=True)
        out[f] = (h.numpy().reshape(n, order="F"), h, torch.empty_like(h, dtype=torch.float32))
    return out


def _read(sv, buffers, single):
    got = {}
    for f, (a, flat, flat32) in buffers.items():
        sv.get(f, out=a)
        got[f] = flat32.copy_(flat) if single else a
    return got


def _open(p, seed, keep):
    """A solver with the fields of ``seed``, and host copies of those named in ``keep``."""
    sv = S.Solver(p)
    kept = {}
    for f, t in fields(p, seed).items():
        a = _host(t)
        sv.set(f, a)
        if f in keep:
            kept[f] = a
    return sv, kept


def _batch_params(case):
    cases = batch.sweep_cases(case["count"], seed=case["draw_seed"], edges=(case["edge_lo"], case["edge_hi"]))
    for p in cases:
        p.init = S.INIT["none"]
        p.vr = min(p.vr, 1e2)
        if p.vpdt <= 0.0:
            p.vpdt = p.l1 / (p.n1 - 1) / 11.0
    return cases


def prepare(case, seed):
    kind = case["kind"]
    step_fields = ("RHO", "ETA", "ETA_INI", "P") + VEL
    if kind == "batch":
        opened = [_open(p, seed + 1000 * i, step_fields) for i, p in enumerate(_batch_params(case))]
        return dict(kind=kind, solvers=[o[0] for o in opened], inputs=[o[1] for o in opened],
                    buffers=[_buffers(o[0].params, VEL + ("P",)) for o in opened], opts=_opts(case))
    p = params(case)
    sv, kept = _open(p, seed, step_fields if kind == "mixed" else ("ETA", "ETA_PL", "P") + VEL if kind == "pt" else ())
    if kind == "pt":  # the checkpoint's stresses: at rest
        kept |= {f: torch.zeros(math.prod(n), dtype=torch.float64, pin_memory=True).numpy().reshape(n, order="F") for f, n in ((f, S.field_dims(p, f)) for f in TAU)}
    s = dict(kind=kind, sv=sv, inputs=kept, k=case["k"], setup=case["setup"])
    if kind in ("pt", "mixed"):
        s["buffers"] = _buffers(p, VEL + ("P", "ETA"))
        s["single"] = p.precision != S.PREC["fp64"]
    if kind == "mixed":
        s["opts"] = _opts(case)
    if kind == "adjoint":
        s["b"] = {"V1": _misfit(p, seed)}
    return s


def _opts(case):
    return dict(tol=1e-14, maxiter=case["k"], nout=100, criterion="residual", inner_rtol=1e-14)


def _misfit(p, seed):
    """Derivative of a surface-velocity misfit: a seeded residual on the outermost interior radial face."""
    g = np.random.default_rng(seed)
    b = np.zeros((p.n1 + 1, p.n2, p.n3), order="F")
    b[p.n1 - 1, 1:-1, 1:-1] = 0.01 * g.standard_normal((p.n2 - 2, p.n3 - 2))
    return b


# ---------------------------------------------------------------------------
# one pass
def run(s):
    kind = s["kind"]
    if kind in ("pt", "mixed"):
        for f, a in s["inputs"].items():
            s["sv"].set(f, a)
        if kind == "mixed":
            s["sv"].solve(**s["opts"])
        elif s["setup"] == "plateau":
            s["sv"].solve(tol=1e-14, maxiter=s["k"], nout=10, criterion="reference_plateau")
        else:
            s["sv"].step(s["k"])
        return _read(s["sv"], s["buffers"], s["single"])
    if kind == "batch":
        for sv, inputs in zip(s["solvers"], s["inputs"]):
            for f, a in inputs.items():
                sv.set(f, a)
        S.solve_batch(s["solvers"], S.make_opts(**s["opts"]))
        return [_read(sv, b, True) for sv, b in zip(s["solvers"], s["buffers"])]
    lam, _ = adjoint.adjoint_solve(s["sv"], s["b"], tol=1e-14, maxiter=s["k"], nout=s["k"])
    g = adjoint.vjp(s["sv"], lam)
    g_ini, g_n = adjoint.law_vjp(s["sv"])
    return {"lam": lam, "vjp": g, "g_ini": g_ini, "g_n": np.float64(g_n)}


# ---------------------------------------------------------------------------
# work
def work(case):
    """Bytes: per iteration every field of the scheme read once and, where it changes, written once (26 fields,
    SphericalStokes_diapir.jl:447; transposed iteration: 4 adjoints, 6 memories, 4 right-hand sides, V, η, ηSM and
    the step), and the copies of the pass; flops: of the stencils, about 230 per cell and iteration."""
    if case["kind"] == "batch":
        cells = sum(p.n1 * p.n2 * p.n3 for p in _batch_params(case))
        return {"bytes": cells * (104.0 * case["k"] + 11 * 8.0), "flops": 230.0 * cells * case["k"]}
    cells = case["n1"] * case["n2"] * case["n3"]
    if case["kind"] == "adjoint":
        return {"bytes": cells * 8.0 * (30.0 * case["k"] + 11), "flops": 300.0 * cells * case["k"]}
    word = 4.0 if case["kind"] == "mixed" or case.get("precision") == "fp32" else 8.0
    up = 7 if case["kind"] == "mixed" else 12
    return {"bytes": cells * (26 * word * case["k"] + 8.0 * (up + 5)), "flops": 230.0 * cells * case["k"]}


# ---------------------------------------------------------------------------
# 64-bit values
class Model:
    """The discrete scheme in torch float64: arrays A[i, j, k], i along x1."""

    def __init__(self, p, dev="cuda"):
        self.p = p
        self.sph, self.cyl, self.cart = p.geometry == 0, p.geometry == 1, p.geometry == 2
        self.x = _axes(p, dev)
        self.d1, self.d2, self.d3 = (p.n1 - 1) / p.l1, (p.n2 - 1) / p.l2, (p.n3 - 1) / p.l3
        one, zero = torch.ones((), dtype=torch.float64, device=dev), torch.zeros((), dtype=torch.float64, device=dev)
        x1, x2 = self.x[0].view(-1, 1, 1), self.x[1].view(1, -1, 1)
        half = lambda a, dim: 0.5 * (a.narrow(dim, 0, a.shape[dim] - 1) + a.narrow(dim, 1, a.shape[dim] - 1))  # noqa: E731
        ones1, ones2 = torch.ones_like(x1), torch.ones_like(x2)
        self.iR, self.iRh = (1 / x1, 1 / half(x1, 0)) if not self.cart else (ones1, ones1[1:])
        if self.sph:
            h = half(x2, 1)
            self.iS, self.iSh, self.ct, self.cth = 1 / torch.sin(x2), 1 / torch.sin(h), 1 / torch.tan(x2), 1 / torch.tan(h)
            self.iR3, self.iRh3 = self.iR, self.iRh
        else:
            self.iS, self.iSh, self.ct, self.cth = ones2, ones2[:, 1:], 0 * ones2, 0 * ones2[:, 1:]
            self.iR3, self.iRh3 = ones1, ones1[1:]
        self.one, self.zero = one, zero
        self.kbc = p.dmp * 2.0 * math.pi * p.vpdt / p.l_ref
        self.gsc = 4.0 * math.pi * p.vpdt / p.l_ref
        self.traction, self.fs = p.bc == S.BC["stress"], p.bc == S.BC["free_surface"]

    # strain rates: divergence, three normal rates at cells, three engineering shear rates at edges
    def strain(self, V):
        V1, V2, V3 = V
        n1, n2, n3 = self.p.n1, self.p.n2, self.p.n3
        a, b, c = V1.diff(dim=0) * self.d1, V2.diff(dim=1) * self.d2 * self.iR, V3.diff(dim=2) * self.d3 * self.iR3 * self.iS
        ax, ay = 0.5 * (V1[1:] + V1[:-1]), 0.5 * (V2[:, 1:] + V2[:, :-1])
        if self.sph:
            div = a + b + c + 2 * self.iR * ax + self.ct * self.iR * ay
            t = div / 3
            D = (a - t, b + self.iR * ax - t, c + self.iR * ax + self.ct * self.iR * ay - t)
        elif self.cyl:
            div = a + b + c + self.iR * ax
            t = div / 3
            D = (a - t, b + self.iR * ax - t, c - t)
        else:
            div, D = a + b + c, (a, b, c)
        v2, v1 = V2[:, 1:n2, 1:-1], V1[1:n1, :, 1:-1]
        E12 = v2.diff(dim=0) * self.d1 + self.iRh * v1.diff(dim=1) * self.d2
        if not self.cart:
            E12 = E12 - 0.5 * (v2[1:] + v2[:-1]) * self.iRh
        v3, v1 = V3[:, 1:-1, 1:n3], V1[1:n1, 1:-1, :]
        E13 = v3.diff(dim=0) * self.d1 + self.iRh3 * self.iS[:, 1:-1] * v1.diff(dim=2) * self.d3
        if self.sph:
            E13 = E13 - 0.5 * (v3[1:] + v3[:-1]) * self.iRh
        v3, v2 = V3[1:-1, :, 1:n3], V2[1:-1, 1:n2, :]
        E23 = self.iR[1:-1] * v3.diff(dim=1) * self.d2 + self.iR3[1:-1] * self.iSh * v2.diff(dim=2) * self.d3
        if self.sph:
            E23 = E23 - 0.5 * (v3[:, 1:] + v3[:, :-1]) * self.iR[1:-1] * self.cth
        return div, D, (E12, E13, E23)

    @staticmethod
    def edges(a):
        """Sums over the four cells around each edge."""
        s12, s13, s23 = a[:, :, 1:-1], a[:, 1:-1, :], a[1:-1]
        return (s12[1:, 1:] + s12[1:, :-1] + s12[:-1, 1:] + s12[:-1, :-1], s13[1:, :, 1:] + s13[1:, :, :-1] + s13[:-1, :, 1:] + s13[:-1, :, :-1],
                s23[:, 1:, 1:] + s23[:, 1:, :-1] + s23[:, :-1, 1:] + s23[:, :-1, :-1])

    # momentum residuals at the interior nodes from σ (cells) and the edge stresses
    def momentum(self, s, T, rho=None):
        s11, s22, s33 = s
        T12, T13, T23 = T
        av = lambda a, dim: 0.5 * (a.narrow(dim, 1, a.shape[dim] - 1) + a.narrow(dim, 0, a.shape[dim] - 1))  # noqa: E731
        a1, a2, a3 = (x[:, 1:-1, 1:-1] for x in s)
        r1 = a1.diff(dim=0) * self.d1 + self.iRh * T12.diff(dim=1) * self.d2 + self.iRh3 * self.iS[:, 1:-1] * T13.diff(dim=2) * self.d3
        if self.sph:
            r1 = r1 + (2 * av(a1, 0) - av(a2, 0) - av(a3, 0)) * self.iRh + av(T12, 1) * self.iRh * self.ct[:, 1:-1]
        elif self.cyl:
            r1 = r1 + (av(a1, 0) - av(a2, 0)) * self.iRh
        a2, a3 = s22[1:-1, :, 1:-1], s33[1:-1, :, 1:-1]
        iR = self.iR[1:-1]
        r2 = T12.diff(dim=0) * self.d1 + iR * a2.diff(dim=1) * self.d2 + self.iR3[1:-1] * self.iSh * T23.diff(dim=2) * self.d3
        if self.sph:
            r2 = r2 + 3 * av(T12, 0) * iR + (av(a2, 1) - av(a3, 1)) * iR * self.cth
        elif self.cyl:
            r2 = r2 + 2 * av(T12, 0) * iR
        a3 = s33[1:-1, 1:-1]
        r3 = T13.diff(dim=0) * self.d1 + iR * T23.diff(dim=1) * self.d2 + self.iR3[1:-1] * self.iS[:, 1:-1] * a3.diff(dim=2) * self.d3
        if self.sph:
            r3 = r3 + 3 * av(T13, 0) * iR + 2 * av(T23, 1) * iR * self.ct[:, 1:-1]
        elif self.cyl:
            r3 = r3 + av(T13, 0) * iR
        if rho is not None:
            if self.cart:
                r3 = r3 - self.p.g * av(rho[1:-1, 1:-1], 2)
            else:
                r1 = r1 - self.p.g * av(rho[:, 1:-1, 1:-1], 0)
        return r1, r2, r3

    def add_interior(self, V, dV):
        V = [v.clone() for v in V]
        V[0][1:-1, 1:-1, 1:-1] += dV[0]
        V[1][1:-1, 1:-1, 1:-1] += dV[1]
        V[2][1:-1, 1:-1, 1:-1] += dV[2]
        return V

    # boundary velocities, face pair by face pair; homog: the correction's (no boundary data)
    def bc(self, V, homog):
        p = self.p
        V = [v.clone() for v in V]

        def ghost(f, dim, kind, sides=(0, 1)):
            v = V[f]
            n = v.shape[dim]
            for side in sides:
                b, i = (0, 1) if side == 0 else (n - 1, n - 2)
                src, dst = v.select(dim, i).clone(), v.select(dim, b)
                if kind == "neg":
                    dst.copy_(-src)
                elif kind == "copy":
                    dst.copy_(src)
                elif kind == "zero" or (homog and kind == "lin"):
                    dst.zero_()
                else:
                    x2 = self.x[1]
                    c, rate = (math.pi / 2, p.r * p.sh) if self.sph else (0.0, p.r * p.sh) if self.cyl else (0.0, p.sh)
                    line = ((x2 - c) * rate)
                    if dim == 1:
                        value = line[0 if side == 0 else -1].expand_as(src)
                    elif dim == 0:
                        value = line.view(-1, 1).expand_as(src)
                    else:
                        value = line.view(1, -1).expand_as(src)
                    dst.copy_(value if kind == "lin" else (-src if homog else 2 * value - src))

        def divfree(f, dim, sides=(0, 1)):
            # the normal ghost that makes the boundary cells divergence-free
            n = V[f].shape[dim]
            for side in sides:
                old = V[f].select(dim, 0 if side == 0 else n - 1)
                cell, sign = (0, -1.0) if side == 0 else (n - 2, 1.0)
                W = [v.narrow(dim, cell, 2 if i == f else 1) for i, v in enumerate(V)]
                inner = W[f].narrow(dim, 1 if side == 0 else 0, 1)
                sl = lambda a: a.narrow(dim, cell, 1) if a.shape[dim] > 1 else a  # noqa: E731
                iR, iR3, iS, ct = (sl(a) for a in (self.iR, self.iR3, self.iS, self.ct))
                c1 = (2 if self.sph else 1) * iR
                coef = (self.d1 + 0 * iR, self.d2 * iR, self.d3 * iR3 * iS)
                mean = (0.5 * c1, 0.5 * ct * iR, 0 * iR)
                total = 0.0
                for i in range(3):
                    if i == f:
                        total = total + (-sign * coef[i] + mean[i]) * inner
                    else:
                        hi, lo = W[i].narrow(i, 1, W[i].shape[i] - 1), W[i].narrow(i, 0, W[i].shape[i] - 1)
                        total = total + coef[i] * (hi - lo) + mean[i] * (hi + lo)
                old.copy_((-total / (sign * coef[f] + mean[f])).squeeze(dim))

        if p.bc == S.BC["free_slip"] or self.fs:
            ghost(0, 0, "neg", (0,) if self.fs else (0, 1)); ghost(1, 0, "copy"); ghost(2, 0, "copy")
            if self.fs:
                divfree(0, 0, (1,))
            ghost(0, 1, "copy"); ghost(1, 1, "neg"); ghost(2, 1, "copy")
            ghost(0, 2, "copy"); ghost(1, 2, "copy"); ghost(2, 2, "neg")
        elif self.traction:
            ghost(0, 0, "neg"); ghost(1, 0, "copy"); ghost(2, 0, "copy")
            ghost(0, 1, "copy"); ghost(2, 1, "copy"); divfree(1, 1)
            ghost(0, 2, "copy"); ghost(1, 2, "copy"); divfree(2, 2)
        elif not self.cart:
            ghost(0, 0, "neg"); ghost(1, 0, "copy"); ghost(2, 0, "copy")
            ghost(0, 1, "zero"); ghost(1, 1, "neg"); ghost(2, 1, "lin")
            ghost(0, 2, "zero"); ghost(1, 2, "zero"); ghost(2, 2, "lin2")
        else:
            ghost(0, 0, "lin2"); ghost(1, 0, "zero"); ghost(2, 0, "zero")
            ghost(0, 1, "lin"); ghost(1, 1, "neg"); ghost(2, 1, "zero")
            ghost(0, 2, "copy"); ghost(1, 2, "copy"); ghost(2, 2, "neg")
        return V

    @staticmethod
    def spread(a):
        """Interior cells -> all cells: boundary cells take the value of the nearest interior cell."""
        for dim in range(3):
            a = torch.cat((a.narrow(dim, 0, 1), a, a.narrow(dim, a.shape[dim] - 1, 1)), dim)
        return a

    def keep_rims(self, a, old):
        """The Cartesian script copies face interiors only: edges and corners keep their value."""
        if not self.cart:
            return a
        on = [torch.zeros(n, dtype=torch.int64, device=a.device) for n in a.shape]
        for o in on:
            o[0] = o[-1] = 1
        rim = (on[0].view(-1, 1, 1) + on[1].view(1, -1, 1) + on[2].view(1, 1, -1)) >= 2
        return torch.where(rim, old, a)

    def maxloc(self, eta):
        m, c = eta, slice(1, -1)
        for dim in range(3):
            at = [c, c, c]
            for cut in (slice(0, -2), slice(2, None)):
                at[dim] = cut
                inner = m[c, c, c] if m is eta else m
                m = torch.maximum(inner, eta[tuple(at)])
        return self.keep_rims(self.spread(m), eta)

    def pressure(self, P, D_or_tau, V, load):
        """Boundary pressures that a prescribed normal stress fixes."""
        t11, t22, t33 = D_or_tau
        if self.traction:
            P = P.clone()
            s2, s3 = self.sig
            both = 0.5 * ((t22 - s2) + (t33 - s3))
            for j in (0, -1):
                P[:, j] = (t22 - s2)[:, j]
            for k in (0, -1):
                P[:, :, k] = (t33 - s3)[:, :, k]
                for j in (0, -1):
                    P[:, j, k] = both[:, j, k]
        if self.fs:
            P = P.clone()
            P[-1] = t11[-1] + load[-1] + self.p.fs_kappa * 0.5 * (V[0][-2] + V[0][-1])
        return P

    sig = (0.0, 0.0)

    def sweep(self, st, eta, sm, rP=0.0, rV=(0.0, 0.0, 0.0), rho=None, load=None, law=None, homog=False):
        """One PT iteration of the state [P, V, τ normal, τ shear]; returns it and the step's η."""
        P, V, t, T = st
        div, D, E = self.strain(V)
        gs, kb = self.gsc * sm, self.kbc * sm
        f = eta / (eta + gs)
        P = P - kb * (div + rP)
        t = [(a + 2 * gs * d) * f for a, d in zip(t, D)]
        T = [(a + 0.25 * self.gsc * s * e) * h / (h + self.gsc * s) for a, s, h, e in zip(T, self.edges(sm), self.edges(eta), E)]
        P = self.pressure(P, t, V, load)
        dt = self.p.vpdt ** 2 / (kb + gs * f)
        if law is not None:
            eta = law(eta, D, E, t, T)
        r = self.momentum([a - P for a in t], T, rho)
        i = slice(1, -1)
        steps = (0.5 * (dt[1:, i, i] + dt[:-1, i, i]), 0.5 * (dt[i, 1:, i] + dt[i, :-1, i]), 0.5 * (dt[i, i, 1:] + dt[i, i, :-1]))
        V = self.bc(self.add_interior(V, [(a + b) * s for a, b, s in zip(r, rV, steps)]), homog)
        return [P, V, t, T], eta

    def shear(self, E):
        """Means of the shear edges around each interior cell."""
        e12, e13, e23 = E
        return (0.25 * (e12[1:, 1:] + e12[1:, :-1] + e12[:-1, 1:] + e12[:-1, :-1]), 0.25 * (e13[1:, :, 1:] + e13[1:, :, :-1] + e13[:-1, :, 1:] + e13[:-1, :, :-1]),
                0.25 * (e23[:, 1:, 1:] + e23[:, 1:, :-1] + e23[:, :-1, 1:] + e23[:, :-1, :-1]))

    def edot_eta(self, D, E, eta_ini, phase, n_exp=None):
        """Target viscosity of the strain-rate power law."""
        n = self.p.n_exp if n_exp is None else n_exp
        i = slice(1, -1)
        a, b, c = self.shear(E)
        ed = self.spread(torch.sqrt(0.5 * sum(d[i, i, i] ** 2 for d in D) + 0.25 * (a * a + b * b + c * c)))
        pl = eta_ini * (ed / self.p.edot_bg) ** ((1 - n) / n)
        return torch.where(phase > 0, eta_ini, 2 / (1 / eta_ini + 1 / pl))

    def laws(self, f):
        """η after a stress update, for the viscosity law of the parameters."""
        p, rheo = self.p, S.RHEO
        i = slice(1, -1)
        ini, phase = f["ETA_INI"], f["PHASE"]
        if p.rheology == rheo["linear"]:
            return None
        if p.rheology == rheo["edot_power_relax"]:
            return lambda eta, D, E, t, T: torch.exp((1 - p.relax) * torch.log(eta) + p.relax * torch.log(self.edot_eta(D, E, ini, phase)))
        hold = {"pl": f.get("ETA_PL"), "tii": torch.zeros_like(ini)}
        ne = torch.where(phase > 0, self.one, self.one * p.n_exp)

        def tau_law(eta, D, E, t, T):
            a, b, c = self.shear(T)
            tii = torch.sqrt(0.5 * sum(x[i, i, i] ** 2 for x in t) + a * a + b * b + c * c)
            hold["tii"] = tii = self.keep_rims(self.spread(tii), hold["tii"])
            pl = ini * (tii / p.tau_C) ** (1 - ne)
            if p.rheology == rheo["tau_power_relax"]:
                if p.n_exp <= 1.0:
                    return eta
                hold["pl"] = pl = torch.exp(torch.log(pl) * p.relax + torch.log(hold["pl"]) * (1 - p.relax))
            return 2 / (1 / ini + 1 / pl)

        return tau_law

    def rest(self):
        """Zero stresses."""
        p = self.p
        z = lambda *n: torch.zeros(n, dtype=torch.float64, device=self.x[0].device)  # noqa: E731
        return ([z(p.n1, p.n2, p.n3) for _ in range(3)],
                [z(p.n1 - 1, p.n2 - 1, p.n3 - 2), z(p.n1 - 1, p.n2 - 2, p.n3 - 1), z(p.n1 - 2, p.n2 - 1, p.n3 - 1)])

    def iterate(self, f, k):
        st, eta = [f["P"], [f[v] for v in VEL], *self.rest()], f["ETA"]
        law = self.laws(f)
        self.sig = (self.p.sig_bc[1], self.p.sig_bc[2])
        for _ in range(k):
            st, eta = self.sweep(st, eta, self.maxloc(eta), rho=f["RHO"], load=f.get("TOP_LOAD"), law=law)
        return dict(zip(VEL, st[1])) | {"P": st[0], "ETA": eta}

    def residual(self, f, V, P, eta):
        """η, boundary velocities and pressure, and the residual of the Stokes equations."""
        self.sig = (self.p.sig_bc[1], self.p.sig_bc[2])
        if self.p.rheology == S.RHEO["edot_power_relax"]:
            _, D, E = self.strain(V)
            eta = self.edot_eta(D, E, f["ETA_INI"], f["PHASE"])
        V = self.bc(V, False)
        div, D, E = self.strain(V)
        t = [2 * eta * d for d in D]
        T = [0.25 * h * e for h, e in zip(self.edges(eta), E)]
        Pb = self.pressure(P, t, V, f.get("TOP_LOAD"))
        return V, Pb, eta, div, self.momentum([a - Pb for a in t], T, f["RHO"])

    def correct(self, f, k):
        """One defect-correction step of k sweeps from the given velocities and pressure."""
        V, P, eta = [f[v] for v in VEL], f["P"], f["ETA"]
        V, _, eta, rP, rV = self.residual(f, V, P, eta)
        sm = self.maxloc(eta)
        st = [torch.zeros_like(P), [torch.zeros_like(v) for v in V], *self.rest()]
        self.sig = (0.0, 0.0)
        load = torch.zeros_like(P) if self.fs else None
        for _ in range(k):
            st, _ = self.sweep(st, eta, sm, rP=rP, rV=rV, load=load, homog=True)
        V, P = [a + b for a, b in zip(V, st[1])], P + st[0]
        V, Pb, eta, _, _ = self.residual(f, V, P, eta)
        return dict(zip(VEL, V)) | {"P": Pb if self.traction else P, "ETA": eta}

    def transposed(self, f, b1, k):
        """k iterations of the transposed scheme for the right-hand side b1 on V1, then the gradients of λᵀR."""
        p = self.p
        V = [f[v] for v in VEL]
        _, D, E = self.strain(V)
        law = p.rheology == S.RHEO["edot_power_relax"]
        eta = self.edot_eta(D, E, f["ETA_INI"], f["PHASE"]) if law else f["ETA"]
        sm = self.maxloc(eta)
        gs, kb = self.gsc * sm, self.kbc * sm
        i = slice(1, -1)
        dt = p.vpdt ** 2 / (kb + gs * (eta / (eta + gs)))
        steps = (0.5 * (dt[1:, i, i] + dt[:-1, i, i]), 0.5 * (dt[i, 1:, i] + dt[i, :-1, i]), 0.5 * (dt[i, i, 1:] + dt[i, i, :-1]))
        aE, aG = [0.25 * s for s in self.edges(eta)], [0.25 * s for s in self.edges(gs)]
        self.sig = (0.0, 0.0)
        # stresses (and pressure) -> momentum rows, linear; velocities -> stresses and divergence, at the state
        t = [a.requires_grad_() for a in self.rest()[0]]
        T = [a.requires_grad_() for a in self.rest()[1]]
        P = torch.zeros_like(eta).requires_grad_()
        Pb = self.pressure(P, t, V, None)
        rows = self.momentum([a - Pb for a in t], T)
        X = [torch.zeros_like(v).requires_grad_() for v in V]
        W = [v + x for v, x in zip(V, self.bc(X, True))]
        ini, n_exp = f["ETA_INI"].clone().requires_grad_(), (self.one * p.n_exp).requires_grad_()
        div, D, E = self.strain(W)
        free = self.edot_eta(D, E, ini, f["PHASE"], n_exp) if law else eta.clone().requires_grad_()
        out = [2 * free * d for d in D] + [0.25 * h * e for h, e in zip(self.edges(free), E)] + [div]
        lV = [torch.zeros_like(x[i, i, i]) for x in X]
        lP, mu = torch.zeros_like(eta), [torch.zeros_like(o) for o in out[:6]]
        rate = [gs / (eta + gs)] * 3 + [g / (e + g) for g, e in zip(aG, aE)]
        stiff = [2 * eta] * 3 + aE
        b = [b1[i, i, i], 0.0, 0.0]
        for _ in range(k):
            got = torch.autograd.grad(rows, t + T + [P], lV, retain_graph=True)
            lP = lP - kb * got[6]
            mu = [m + w * (s * a - m) for m, w, s, a in zip(mu, rate, stiff, got)]
            aV = torch.autograd.grad(out, X, [m / s for m, s in zip(mu, stiff)] + [lP], retain_graph=True)
            lV = [l + s * (a[i, i, i] - c) for l, s, a, c in zip(lV, steps, aV, b)]
        got = torch.autograd.grad(rows, t + T + [P], lV, retain_graph=True)
        want = X + [free] + ([ini, n_exp] if law else [])
        g = torch.autograd.grad(out, want, list(got[:6]) + [lP], retain_graph=True)
        rho = torch.zeros_like(eta).requires_grad_()
        weight = [(r, l) for r, l in zip(self.momentum([torch.zeros_like(eta)] * 3, self.rest()[1], rho), lV) if r.requires_grad]
        g_rho = torch.autograd.grad([r for r, _ in weight], rho, [l for _, l in weight])[0]
        pad = torch.nn.functional.pad
        whole = lambda parts: {v: pad(a, (1, 1, 1, 1, 1, 1)) for v, a in zip(VEL, parts)}  # noqa: E731
        return {"lam": whole(lV) | {"P": lP},
                "vjp": whole([a[i, i, i] for a in g[:3]]) | {"P": got[6], "ETA": g[3], "RHO": g_rho},
                "g_ini": g[4] if law else g[3], "g_n": g[5] if law else self.zero}


def _out(v, single):
    """A field as ``run`` hands it on: FP32 results as one run of values in the solver's order."""
    return v.permute(2, 1, 0).reshape(-1) if single else v.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        got = []
        for i, p in enumerate(_batch_params(case)):
            r = Model(p).correct(fields(p, seed + 1000 * i), case["k"])
            got.append({f: _out(r[f], True) for f in VEL + ("P",)})
        return got
    p = params(case)
    f, m = fields(p, seed), Model(p)
    if kind == "pt" or kind == "mixed":
        single = p.precision != S.PREC["fp64"]
        r = m.iterate(f, case["k"]) if kind == "pt" else m.correct(f, case["k"])
        return {name: _out(r[name], single) for name in VEL + ("P", "ETA")}
    r = m.transposed(f, torch.from_numpy(_misfit(p, seed)).cuda(), case["k"])
    return {a: {n: v.detach() for n, v in x.items()} if isinstance(x, dict) else x.detach() for a, x in r.items()}
