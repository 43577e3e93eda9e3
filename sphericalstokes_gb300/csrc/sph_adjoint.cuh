// Adjoint (vector-Jacobian product) kernels of the FP64 Stokes residual.
// Forward map (residual64 of sphstokes.cu):
//   V (all entries) --strain rates, 2ηD / avg4(η)D--> τ  (k_cells)
//   σ_ii = τ_ii - P_eff, P_eff = P or τ_nn - σ_bc on far-field-stress boundary cells
//   R_V = momentum(σ, τ_edges) - ρg at interior nodes  (k_nodes)
//   R_P = div V at every cell
// and, for the interior-unknown form, V = B(V_interior) by the homogeneous BC program; under the
// strain-rate law η depends on V as well.
//
// Transposed PT with the forward scheme's stress memory: the forward PT relaxes τ toward 2η E(V) at
// the rate 1 - f (f = η/(η + GSDT); edges: avg4 η, avg4 GSDT) and drives V with the momentum of
// τ.  The transposed iteration relaxes the memory μ toward 2η M_τᵀ λ_V at the same rate and drives
// λ_V with Eᵀ μ: the coupling products are the transposes of the forward ones.
//
// Every kernel gathers: a thread owns the entries it writes and reads the adjoints that reach them, so
// there are no atomics and no clearing of accumulators; but for the transposed stress ghosts
// (k_bc_adjoint, BC_STRESS), which scatter to neighbours with FP64 atomics.  The kernels march along x3 like those of
// sph_march.cuh and are bound the same way, by FP64 instructions; the factors that stay fixed
// during a solve (rates, stiffnesses, the state's strain rates, the law's
// derivative) are made once by k_adj_setup.
//   k_adj_stress   λ_V -> adjoint of σ, τ (cells, edges), of P; MEM: μ and λ_P updated
//   k_adj_eta      per cell λᵀ ∂R/∂η (and, for the law, that times dη_t/dε̇)
//   k_adj_collect, k_adj_law   the law's dependence on V added to the adjoints of the strain rates
//   k_adj_strain   adjoints of strain rates and div V -> V (all entries)
// Measured on a GB300, 63^3 sector under the strain-rate law: 118 us per transposed iteration (820 with
// scatters by FP64 atomics and coefficients evaluated as stencils of unit vectors), the FP64 units 56 - 77 %
// busy in the cell and node kernels; the rest is the five BC stages and launches.
#pragma once
#include "sph_march.cuh"
#include "sph_pt.cuh"

namespace sph {

struct Adj {
    const double *lV1, *lV2, *lV3;       // adjoint of the momentum rows (interior nodes)
    double* lP;                          // adjoint of the continuity rows
    const double* bP;                    // MEM: right-hand side of the P equations
    double *d11, *d22, *d33;             // adjoint of the strain rates: 2η aτ, or the memory μ (MEM)
    double *e12, *e13, *e23;             // edges: avg4(η) aτ, or μ
    double *x12, *x13, *x23;             // law: edge adjoints with the law's part
    double *q12, *q13, *q23;             // edges' share of λᵀ ∂R/∂η of each of their four cells
    double *E1, *M1, *E2, *M2, *E3;      // cells: what V reads of them (cell_out)
    double *aV1, *aV2, *aV3, *aP;        // output: adjoint of V (all entries), P
    double *gEta, *gRho, *gW;            // λᵀ ∂R/∂η, λᵀ ∂R/∂ρ per cell; gEta times the law's derivative
    // fixed factors (k_adj_setup)
    double *wc, *ie;                     // cells: 1 - f, 1 / η
    double *y12, *y13, *y23, *w12, *w13, *w23;  // edges: avg4 η, 1 - f
    double *c11, *c22, *c33;             // D_ii
    double *g12, *g13, *g23;             // law: D_edge / (4 avg4 η)
    double *lw, *lr, *la, *lb, *lc;      // law: dη_t/dε̇, 1/(2ε̇), and (mean shear rates) / (16 ε̇) of interior cells
};

// cell adjoints aD_ii and λ_P as the six face velocities read them: +-E1 + M1 (V1), +-E2 + M2, +-E3
template <int G>
__device__ __forceinline__ void cell_out(const CellMetric<double>& m, double d1, const Adj& a, int c, double D11, double D22, double D33, double lP) {
    const double q = G == CART ? lP : fma(-1.0 / 3.0, D11 + D22 + D33, lP);
    a.E1[c] = (q + D11) * d1;
    a.E2[c] = (q + D22) * m.a2;
    a.E3[c] = (q + D33) * m.a3;
    if (G != CART) a.M1[c] = 0.5 * fma(m.c1, q, G == SPH ? m.e1 * (D22 + D33) : m.e1 * D22);
    if (G == SPH) a.M2[c] = 0.5 * fma(m.c2, q, m.e2 * D33);
}

// factors that stay fixed for a state: from V, η, ηSM, and for the law sDD and the edge shear rates of k_cells
template <int G, bool LAW>
__global__ void __launch_bounds__(MC_NT) k_adj_setup(const __grid_constant__ KP<double> p, const __grid_constant__ Adj a) {
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x, k = blockIdx.y;
    const int i = col % d.n1, j = col / d.n1;
    if (j >= d.n2) return;
    const int sy = d.sy, sz = d.sz, c = i + sy * j + sz * k;
    const double et = p.eta[c], gs = p.gsc * p.etaSM[c];
    a.wc[c] = gs / (et + gs);
    a.ie[c] = 1.0 / et;
    const CellD<double> D = cell_strain<double, G>(p.geo, p.d1, p.d2, p.d3, i, j, p.V1[c], p.V1[c + 1], p.V2[c], p.V2[c + sy], p.V3[c], p.V3[c + sz]);
    a.c11[c] = D.D11; a.c22[c] = D.D22; a.c33[c] = D.D33;
    auto edge = [&](double* y, double* w, double* g, int q, int o1, int o2, int o3, double De) {
        const double aE = 0.25 * (p.eta[q] + p.eta[q + o1] + p.eta[q + o2] + p.eta[q + o3]);
        const double aG = 0.25 * p.gsc * (p.etaSM[q] + p.etaSM[q + o1] + p.etaSM[q + o2] + p.etaSM[q + o3]);
        y[c] = aE;
        w[c] = aG / (aE + aG);
        if (LAW) g[c] = 0.25 * De / aE;
    };
    if (i < d.n1 - 1 && j < d.n2 - 1 && k < d.n3 - 2) {
        const int q = c + sz;
        edge(a.y12, a.w12, a.g12, q, sy, 1, 1 + sy, edge12<double, G>(p.geo, p.d1, p.d2, i, p.V2[q + sy], p.V2[q + sy + 1], p.V1[q + 1], p.V1[q + 1 + sy]));
    }
    if (i < d.n1 - 1 && j < d.n2 - 2 && k < d.n3 - 1) {
        const int q = c + sy;
        edge(a.y13, a.w13, a.g13, q, sz, 1, 1 + sz, edge13<double, G>(p.geo, p.d1, p.d3, i, j, p.V3[q + sz], p.V3[q + sz + 1], p.V1[q + 1], p.V1[q + 1 + sz]));
    }
    if (i < d.n1 - 2 && j < d.n2 - 1 && k < d.n3 - 1) {
        const int q = c + 1;
        edge(a.y23, a.w23, a.g23, q, sz, sy, sy + sz, edge23<double, G>(p.geo, p.d2, p.d3, i, j, p.V3[q + sz], p.V3[q + sz + sy], p.V2[q + sy], p.V2[q + sy + sz]));
    }
    if (!LAW) return;
    // The law (k_edot, unrelaxed target η_t = 2/(1/η_ini + 1/η_PL), η_PL = η_ini (ε̇_II/ε̇_bg)^m, m = (1-n)/n, ε̇_II of the
    // clamped interior cell s from sDD(s) and the 4-edge means a, b, c of the shear rates):
    //   dη_t/dε̇ = m η_t² / (2 η_PL ε̇),  dε̇/dsDD = 1/(2ε̇),  dε̇/da = a/(4ε̇),  da/ds12(edge) = 1/4,  sDD = ½ Σ D_ii²
    const int s = clampi(i, 1, d.n1 - 2) + sy * clampi(j, 1, d.n2 - 2) + sz * clampi(k, 1, d.n3 - 2);
    const int e = s - 1 - sy - sz;
    const double av = 0.25 * (p.s12[e] + p.s12[e + sy] + p.s12[e + 1] + p.s12[e + 1 + sy]);
    const double bv = 0.25 * (p.s13[e] + p.s13[e + sz] + p.s13[e + 1] + p.s13[e + 1 + sz]);
    const double cv = 0.25 * (p.s23[e] + p.s23[e + sz] + p.s23[e + sy] + p.s23[e + sy + sz]);
    const double ed = sqrt(p.sDD[s] + 0.25 * (av * av + bv * bv + cv * cv));
    double w = 0.0;
    if (!(p.phase && p.phase[c]) && ed > 0.0) {
        const double ei = p.eta_ini[c], m = (1.0 - p.n_exp) / p.n_exp;
        const double pl = ei * pow(ed / p.edot_bg, m), t = 2.0 / (1.0 / ei + 1.0 / pl);
        w = m * t * t / (2.0 * pl * ed);
    }
    a.lw[c] = w;
    const bool own = s == c && ed > 0.0;  // interior cell
    a.lr[c] = own ? 1.0 / (2.0 * ed) : 0.0;
    a.la[c] = own ? av / (16.0 * ed) : 0.0;
    a.lb[c] = own ? bv / (16.0 * ed) : 0.0;
    a.lc[c] = own ? cv / (16.0 * ed) : 0.0;
}

// λ_V -> adjoint of σ (cells; the traction-slaved pressure of far-field-stress boundary cells goes to τ22 / τ33)
// and of the edge stresses.  MEM: the memory μ relaxes toward it, μ += (1 - f) (2η σ - μ), whose fixed point is 2η σ
// whatever the rounding of f, and λ_P -= KBDT (M_Pᵀ λ_V - b_P); else the adjoints of the strain rates
// themselves, of P, ρ and η (σ D: no quotient by η, which may be zero).  LAW: k_adj_law finishes the cells.
template <int G, bool MEM, bool LAW>
__global__ void __launch_bounds__(MC_NT) k_adj_stress(const __grid_constant__ KP<double> p, const __grid_constant__ Adj a, int chunk) {
    pdl_enter_small();
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x;
    const int i = col % d.n1, j = col / d.n1;
    if (j >= d.n2) return;
    const int n1 = d.n1, n2 = d.n2, n3 = d.n3, sy = d.sy, sz = d.sz;
    const int k0 = blockIdx.y * chunk, k1 = min(k0 + chunk, n3);
    const double d1 = p.d1;
    const CellMetric<double> m = cell_metric<double, G>(p, i, j);
    // metric factors at the nodes around the cell: 1/x1 at i -+ 1/2, i, i + 1; 1/sin, cot at j, j + 1, j -+ 1/2
    double h0 = 1.0, h1 = 1.0, r0 = 1.0, r1 = 1.0, S0 = 1.0, S1 = 1.0, C0 = 0.0, C1 = 0.0, Th1 = 1.0, K0h = 0.0, K1h = 0.0;
    if (G != CART) {
        h0 = p.geo.invRh[clampi(i - 1, 0, n1 - 2)]; h1 = p.geo.invRh[clampi(i, 0, n1 - 2)];
        r0 = p.geo.invRc[i]; r1 = p.geo.invRc[clampi(i + 1, 0, n1 - 1)];
    }
    if (G == SPH) {
        const int jp = clampi(j + 1, 0, n2 - 1), jm = clampi(j - 1, 0, n2 - 2), jh = clampi(j, 0, n2 - 2);
        S0 = p.geo.invSinC[j]; S1 = p.geo.invSinC[jp]; C0 = p.geo.cotC[j]; C1 = p.geo.cotC[jp];
        Th1 = p.geo.invSinH[jh]; K0h = p.geo.cotH[jm]; K1h = p.geo.cotH[jh];
    }
    const double g1 = G == SPH ? 1.0 : 0.5, hd = 0.5;
    const double c11a = G == CART ? d1 : d1 + g1 * h0, c11b = G == CART ? -d1 : g1 * h1 - d1;
    const double xa = 0.5 * h0, xb = 0.5 * h1, ya = hd * r0 * K0h, yb = hd * r0 * K1h;
    const double r0d2 = r0 * p.d2, z3 = G == SPH ? r0 * S0 * p.d3 : p.d3;
    const double t12a = fma(0.5 * h1, C0, h1 * p.d2), t12b = fma(0.5 * h1, C1, -h1 * p.d2);
    const double u = G == SPH ? 1.5 : (G == CYL ? 1.0 : 0.0), t12c = d1 + u * r0, t12d = u * r1 - d1;
    const double v = G == SPH ? 1.5 : (G == CYL ? 0.5 : 0.0), t13a = G == SPH ? h1 * S1 * p.d3 : p.d3, t13c = d1 + v * r0, t13d = v * r1 - d1;
    const double t23a = G == SPH ? r1 * Th1 * p.d3 : p.d3, t23c = fma(r1, C0, r1 * p.d2), t23d = fma(r1, C1, -r1 * p.d2);
    // interior nodes of the column's neighbours (x1, x2); λ elsewhere does not enter
    const bool i1[2] = {i >= 1, i + 1 <= n1 - 1}, j1[2] = {j >= 1 && j <= n2 - 2, j + 1 <= n2 - 2};
    const bool i2[2] = {i >= 1 && i <= n1 - 2, i + 1 <= n1 - 2}, j2[2] = {j >= 1, j + 1 <= n2 - 1};
    const bool e12 = i < n1 - 1 && j < n2 - 1, e13 = i < n1 - 1 && j < n2 - 2, e23 = i < n1 - 2 && j < n2 - 1;
    for (int k = k0; k < k1; ++k) {
        const int c = i + sy * j + sz * k;
        const bool kc[2] = {k >= 1 && k <= n3 - 2, k + 1 <= n3 - 2}, k3[2] = {k >= 1, k + 1 <= n3 - 1};
        auto L1 = [&](int x, int y, int z) { return i1[x] && j1[y] && kc[z] ? a.lV1[c + x + sy * y + sz * z] : 0.0; };
        auto L2 = [&](int x, int y, int z) { return i2[x] && j2[y] && kc[z] ? a.lV2[c + x + sy * y + sz * z] : 0.0; };
        auto L3 = [&](int x, int y, int z) { return i2[x] && j1[y] && k3[z] ? a.lV3[c + x + sy * y + sz * z] : 0.0; };
        const double A0 = L1(0, 0, 0), A1 = L1(1, 0, 0), B0 = L2(0, 0, 0), B1 = L2(0, 1, 0), Z0 = L3(0, 0, 0), Z1 = L3(0, 0, 1);
        double s11 = fma(c11a, A0, c11b * A1), s22 = r0d2 * (B0 - B1), s33 = z3 * (Z0 - Z1);
        if (G != CART) {
            const double x = fma(xa, A0, xb * A1);
            s22 -= x;
            if (G == SPH) {
                const double y = fma(ya, B0, yb * B1);
                s22 += y;
                s33 -= x + y;
            }
        }
        const double pe = -(s11 + s22 + s33);
        const bool b2 = p.traction && (j == 0 || j == n2 - 1), b3 = p.traction && (k == 0 || k == n3 - 1);
        if (b2 && b3) { s22 += 0.5 * pe; s33 += 0.5 * pe; }
        else if (b2) s22 += pe;
        else if (b3) s33 += pe;
        const double aP = b2 || b3 ? 0.0 : pe;
        double D11, D22, D33, lP = a.lP[c];
        if (MEM) {
            const double w = a.wc[c], e2 = 2.0 * p.eta[c];
            D11 = a.d11[c]; D22 = a.d22[c]; D33 = a.d33[c];
            D11 = fma(w, fma(e2, s11, -D11), D11); D22 = fma(w, fma(e2, s22, -D22), D22); D33 = fma(w, fma(e2, s33, -D33), D33);
            lP = fma(-p.kbc * p.etaSM[c], aP - a.bP[c], lP);
            a.lP[c] = lP;
        } else {
            const double e2 = 2.0 * p.eta[c];
            D11 = e2 * s11; D22 = e2 * s22; D33 = e2 * s33;
            a.aP[c] = aP;
            a.gEta[c] = 2.0 * fma(s11, a.c11[c], fma(s22, a.c22[c], s33 * a.c33[c]));
            if (a.gRho) a.gRho[c] = -0.5 * p.g * (G != CART ? A0 + A1 : Z0 + Z1);
        }
        a.d11[c] = D11; a.d22[c] = D22; a.d33[c] = D33;
        if (!LAW) cell_out<G>(m, d1, a, c, D11, D22, D33, lP);
        auto edge = [&](double* E, double* Q, const double* y, const double* w, const double* g, double t, double De) {
            double x = E[c];
            if (MEM) x = fma(w[c], fma(y[c], t, -x), x);
            else x = y[c] * t;
            E[c] = x;
            if (!MEM) Q[c] = 0.25 * t * De;
            else if (LAW) Q[c] = g[c] * x;
        };
        const double A11 = L1(1, 1, 1), B11 = L2(1, 1, 1), Z11 = L3(1, 1, 1);
        if (e12 && k < n3 - 2) {
            const int q = c + sz;
            const double De = MEM ? 0.0 : edge12<double, G>(p.geo, d1, p.d2, i, p.V2[q + sy], p.V2[q + sy + 1], p.V1[q + 1], p.V1[q + 1 + sy]);
            edge(a.e12, a.q12, a.y12, a.w12, a.g12, fma(t12a, L1(1, 0, 1), fma(t12b, A11, fma(t12c, L2(0, 1, 1), t12d * B11))), De);
        }
        if (e13 && k < n3 - 1) {
            const int q = c + sy;
            const double De = MEM ? 0.0 : edge13<double, G>(p.geo, d1, p.d3, i, j, p.V3[q + sz], p.V3[q + sz + 1], p.V1[q + 1], p.V1[q + 1 + sz]);
            edge(a.e13, a.q13, a.y13, a.w13, a.g13, fma(t13a, L1(1, 1, 0) - A11, fma(t13c, L3(0, 1, 1), t13d * Z11)), De);
        }
        if (e23 && k < n3 - 1) {
            const int q = c + 1;
            const double De = MEM ? 0.0 : edge23<double, G>(p.geo, p.d2, p.d3, i, j, p.V3[q + sz], p.V3[q + sz + sy], p.V2[q + sy], p.V2[q + sy + sz]);
            edge(a.e23, a.q23, a.y23, a.w23, a.g23, fma(t23a, L2(1, 1, 0) - B11, fma(t23c, L3(1, 0, 1), t23d * Z11)), De);
        }
    }
}

// λᵀ ∂R/∂η per cell: the cell's own part (of the memory: μ D / η) and its twelve edges'; times the law's derivative for k_adj_law
template <bool MEM, bool LAW>
__global__ void __launch_bounds__(MC_NT) k_adj_eta(const __grid_constant__ KP<double> p, const __grid_constant__ Adj a, int chunk) {
    pdl_enter_small();
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x;
    const int i = col % d.n1, j = col / d.n1;
    if (j >= d.n2) return;
    const int sy = d.sy, sz = d.sz;
    const int k0 = blockIdx.y * chunk, k1 = min(k0 + chunk, d.n3);
    const bool im = i > 0, jm = j > 0;
    for (int k = k0; k < k1; ++k) {
        const int c = i + sy * j + sz * k;
        const bool km = k > 0;
        // (edge entries outside the edges' extents are zero)
        double g;
        if (MEM) g = fma(a.d11[c], a.c11[c], fma(a.d22[c], a.c22[c], a.d33[c] * a.c33[c])) * a.ie[c];
        else g = a.gEta[c];
        if (km) g += (a.q12[c - sz] + (im ? a.q12[c - 1 - sz] : 0.0)) + (jm ? a.q12[c - sy - sz] + (im ? a.q12[c - 1 - sy - sz] : 0.0) : 0.0);
        if (jm) g += (a.q13[c - sy] + (im ? a.q13[c - 1 - sy] : 0.0)) + (km ? a.q13[c - sy - sz] + (im ? a.q13[c - 1 - sy - sz] : 0.0) : 0.0);
        if (im) g += (a.q23[c - 1] + (jm ? a.q23[c - 1 - sy] : 0.0)) + (km ? a.q23[c - 1 - sz] + (jm ? a.q23[c - 1 - sy - sz] : 0.0) : 0.0);
        a.gEta[c] = g;
        if (LAW) a.gW[c] = g * a.lw[c];
    }
}

// The law: η of a cell follows ε̇ of its clamped interior cell s.  First the interior cells next to the
// boundary collect gW of the boundary cells clamped to them, in place (boundary cells are only read) ...
__global__ void __launch_bounds__(256) k_adj_collect(const __grid_constant__ KP<double> p, const __grid_constant__ Adj a) {
    pdl_enter_small();
    const Dims& d = p.d;
    const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y, z = blockIdx.z;
    const int n1 = d.n1, n2 = d.n2, n3 = d.n3, sy = d.sy, sz = d.sz;
    if (x < 1 || y < 1 || z < 1 || x > n1 - 2 || y > n2 - 2 || z > n3 - 2) return;
    if (x != 1 && y != 1 && z != 1 && x != n1 - 2 && y != n2 - 2 && z != n3 - 2) return;
    double h = 0.0;
    for (int dz = (z == 1 ? -1 : 0); dz <= (z == n3 - 2 ? 1 : 0); ++dz)
        for (int dy = (y == 1 ? -1 : 0); dy <= (y == n2 - 2 ? 1 : 0); ++dy)
            for (int dx = (x == 1 ? -1 : 0); dx <= (x == n1 - 2 ? 1 : 0); ++dx) h += a.gW[x + dx + sy * (y + dy) + sz * (z + dz)];
    a.gW[x + sy * y + sz * z] = h;
}
// ... then s passes it on to the strain rates that form ε̇(s) (the factors of boundary cells are zero)
template <int G>
__global__ void __launch_bounds__(MC_NT) k_adj_law(const __grid_constant__ KP<double> p, const __grid_constant__ Adj a, int chunk) {
    pdl_enter_small();
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x;
    const int i = col % d.n1, j = col / d.n1;
    if (j >= d.n2) return;
    const int n1 = d.n1, n2 = d.n2, n3 = d.n3, sy = d.sy, sz = d.sz;
    const int k0 = blockIdx.y * chunk, k1 = min(k0 + chunk, n3);
    const CellMetric<double> m = cell_metric<double, G>(p, i, j);
    const bool e12 = i < n1 - 1 && j < n2 - 1, e13 = i < n1 - 1 && j < n2 - 2, e23 = i < n1 - 2 && j < n2 - 1;
    for (int k = k0; k < k1; ++k) {
        const int c = i + sy * j + sz * k, q = c + sz;
        const double *H = a.gW;
        const double h = H[c] * a.lr[c];
        cell_out<G>(m, p.d1, a, c, fma(h, a.c11[c], a.d11[c]), fma(h, a.c22[c], a.d22[c]), fma(h, a.c33[c], a.d33[c]), a.lP[c]);
        const int o = sy + 1;
        if (e12 && k < n3 - 2)
            a.x12[c] = a.e12[c] + (fma(H[q], a.la[q], H[q + 1] * a.la[q + 1]) + fma(H[q + sy], a.la[q + sy], H[q + o] * a.la[q + o]));
        if (e13 && k < n3 - 1)
            a.x13[c] = a.e13[c] + (fma(H[c + sy], a.lb[c + sy], H[c + o] * a.lb[c + o]) + fma(H[q + sy], a.lb[q + sy], H[q + o] * a.lb[q + o]));
        if (e23 && k < n3 - 1)
            a.x23[c] = a.e23[c] + (fma(H[c + 1], a.lc[c + 1], H[c + o] * a.lc[c + o]) + fma(H[q + 1], a.lc[q + 1], H[q + o] * a.lc[q + o]));
    }
}

// adjoints of strain rates (cells by cell_out, edges X) and of div V -> V, every entry
template <int G>
__global__ void __launch_bounds__(MC_NT) k_adj_strain(const __grid_constant__ KP<double> p, const __grid_constant__ Adj a, const double* __restrict__ X12,
                                                      const double* __restrict__ X13, const double* __restrict__ X23, int chunk) {
    pdl_enter_small();
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x;
    const int w = d.n1 + 1;
    const int i = col % w, j = col / w;
    if (j > d.n2) return;
    const int n1 = d.n1, n2 = d.n2, n3 = d.n3, sy = d.sy, sz = d.sz;
    const int k0 = blockIdx.y * chunk, k1 = min(k0 + chunk, n3 + 1);
    // edge coefficients at (i - 1 | i, j - 1 | j)
    double h0 = 1.0, h1 = 1.0, r0 = 1.0, S0 = 1.0, T0 = 1.0, K0h = 0.0, K1h = 0.0;
    if (G != CART) {
        h0 = p.geo.invRh[clampi(i - 1, 0, n1 - 2)]; h1 = p.geo.invRh[clampi(i, 0, n1 - 2)];
        r0 = p.geo.invRc[clampi(i, 0, n1 - 1)];
    }
    if (G == SPH) {
        const int jm = clampi(j - 1, 0, n2 - 2), jh = clampi(j, 0, n2 - 2);
        S0 = p.geo.invSinC[clampi(j, 0, n2 - 1)]; T0 = p.geo.invSinH[jm]; K0h = p.geo.cotH[jm]; K1h = p.geo.cotH[jh];
    }
    const double h0d2 = h0 * p.d2, e13 = G == SPH ? h0 * S0 * p.d3 : p.d3, e23 = G == SPH ? r0 * T0 * p.d3 : p.d3;
    const double va = G == CART ? -p.d1 : -p.d1 - 0.5 * h1, vb = G == CART ? p.d1 : p.d1 - 0.5 * h0;  // V2 in τ12, V3 in τ13 (spherical)
    const double v3a = G == SPH ? va : -p.d1, v3b = G == SPH ? vb : p.d1;
    const double za = G == SPH ? -r0 * p.d2 - 0.5 * r0 * K1h : -r0 * p.d2, zb = G == SPH ? r0 * p.d2 - 0.5 * r0 * K0h : r0 * p.d2;  // V3 in τ23
    const bool im = i >= 1, jm = j >= 1, ic = i < n1, jc = j < n2;
    for (int k = k0; k < k1; ++k) {
        const int c = i + sy * j + sz * k;
        const bool km = k >= 1, kc = k < n3;
        // edges of the plane below exist for τ12 where 1 <= k <= n3 - 2, for τ13, τ23 where k >= 1; entries outside are zero
        const double x12 = im && jm && km ? X12[c - 1 - sy - sz] : 0.0;  // (i-1, j-1, k-1)
        const double x13 = im && jm && km ? X13[c - 1 - sy - sz] : 0.0;
        const double x23 = im && jm && km ? X23[c - 1 - sy - sz] : 0.0;
        if (jc && kc) {  // V1: cells (i, j, k), (i - 1, j, k); τ12 (i-1, j-1 | j, k-1); τ13 (i-1, j-1, k-1 | k)
            double s = 0.0;
            if (ic) s = (G != CART ? a.M1[c] : 0.0) - a.E1[c];
            if (im) {
                s += a.E1[c - 1];
                if (G != CART) s += a.M1[c - 1];
                s = fma(h0d2, x12 - (km ? X12[c - 1 - sz] : 0.0), s);
                if (jm) s = fma(e13, x13 - X13[c - 1 - sy], s);
            }
            a.aV1[c] = s;
        }
        if (ic && kc) {  // V2: cells (i, j, k), (i, j - 1, k); τ12 (i | i-1, j-1, k-1); τ23 (i-1, j-1, k-1 | k)
            double s = 0.0;
            if (jc) s = (G == SPH ? a.M2[c] : 0.0) - a.E2[c];
            if (jm) {
                s += a.E2[c - sy];
                if (G == SPH) s += a.M2[c - sy];
                s = fma(va, km ? X12[c - sy - sz] : 0.0, fma(vb, x12, s));
                if (im) s = fma(e23, x23 - X23[c - 1 - sy], s);
            }
            a.aV2[c] = s;
        }
        if (ic && jc) {  // V3: cells (i, j, k), (i, j, k - 1); τ13 (i | i-1, j-1, k-1); τ23 (i-1, j | j-1, k-1)
            double s = kc ? -a.E3[c] : 0.0;
            if (km) {
                s += a.E3[c - sz];
                if (jm) s = fma(v3a, X13[c - sy - sz], fma(v3b, x13, s));
                if (im) s = fma(za, X23[c - 1 - sz], fma(zb, x23, s));
            }
            a.aV3[c] = s;
        }
    }
}

// the η contraction through the law to its prefactor and exponent: g dη_t/dη_ini, g dη_t/dn with
// dη_t/dη_ini = η_t/η_ini, dη_t/dn = -η_t² ln(ε̇/ε̇_bg) / (2 η_PL n²).  Phase cells (linear) have η = η_ini.
__global__ void __launch_bounds__(MC_NT) k_adj_law_params(const __grid_constant__ KP<double> p, const __grid_constant__ Adj a, double* __restrict__ gEI,
                                                          double* __restrict__ gN) {
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x, k = blockIdx.y;
    const int i = col % d.n1, j = col / d.n1;
    if (j >= d.n2) return;
    const int sy = d.sy, sz = d.sz, c = i + sy * j + sz * k;
    const double g = a.gEta[c], ei = p.eta_ini[c];
    if (p.phase && p.phase[c]) {
        gEI[c] = g;
        gN[c] = 0.0;
        return;
    }
    const int s = clampi(i, 1, d.n1 - 2) + sy * clampi(j, 1, d.n2 - 2) + sz * clampi(k, 1, d.n3 - 2);
    const int e = s - 1 - sy - sz;
    const double av = 0.25 * (p.s12[e] + p.s12[e + sy] + p.s12[e + 1] + p.s12[e + 1 + sy]);
    const double bv = 0.25 * (p.s13[e] + p.s13[e + sz] + p.s13[e + 1] + p.s13[e + 1 + sz]);
    const double cv = 0.25 * (p.s23[e] + p.s23[e + sz] + p.s23[e + sy] + p.s23[e + sy + sz]);
    const double ed = sqrt(p.sDD[s] + 0.25 * (av * av + bv * bv + cv * cv));
    const double n = p.n_exp, pl = ei * pow(ed / p.edot_bg, (1.0 - n) / n), et = 2.0 / (1.0 / ei + 1.0 / pl);
    gEI[c] = g * et / ei;
    gN[c] = ed > 0.0 ? -g * et * et * log(ed / p.edot_bg) / (2.0 * pl * n * n) : 0.0;
}

// transpose of one homogeneous BC stage (faces normal to axis D) on the velocity adjoints: each boundary
// entry's adjoint goes back to the entries its value was computed from, then is cleared
// Bound by latency: one warp per block and loads before stores, us a stage (63^3, cold caches): x1 faces 16.4 and 4.2 (blocks of
// 256, each op's load behind the store before), copies 4.4 - 7.9 and 3.6 - 4.0.  An iteration 131 and 114, at 39 x 23 x 31 38 and 29.
template <int G, int D>
__global__ void k_bc_adjoint(const __grid_constant__ KP<double> p, const __grid_constant__ Adj a, const __grid_constant__ BcStage st) {
    pdl_enter_small();
    const int u = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y * blockDim.y + threadIdx.y;
    const Dims& d = p.d;
    const int sy = d.sy, sz = d.sz;
    const int step = D == 0 ? 1 : (D == 1 ? sy : sz);
    const int base = D == 0 ? u * sy + v * sz : (D == 1 ? u + v * sz : u + v * sy);
    auto field = [&](int f) { return f == 0 ? a.aV1 : (f == 1 ? a.aV2 : a.aV3); };
    auto ext = [&](int f, int ax) { return (ax == 0 ? d.n1 : (ax == 1 ? d.n2 : d.n3)) + (f == ax); };
    auto on = [&](int f) { return u < ext(f, D == 0 ? 1 : 0) && v < ext(f, D == 2 ? 1 : 2); };
    if (st.op[0].kind != BC_STRESS) {
        // each face point has a source of its own, and the ops are on different fields: all loads, then all stores
        double g[3][2], t[3][2];
#pragma unroll
        for (int o = 0; o < 3; ++o)
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const int f = st.op[o].field, e = ext(f, D);
                if (o >= st.nops || !on(f) || (st.op[o].side >= 0 && st.op[o].side != side)) continue;
                g[o][side] = field(f)[base + (side == 0 ? 0 : e - 1) * step];
                t[o][side] = field(f)[base + (side == 0 ? 1 : e - 2) * step];
            }
#pragma unroll
        for (int o = 0; o < 3; ++o)
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const int f = st.op[o].field, e = ext(f, D), kind = st.op[o].kind;
                if (o >= st.nops || !on(f) || (st.op[o].side >= 0 && st.op[o].side != side)) continue;
                field(f)[base + (side == 0 ? 0 : e - 1) * step] = 0.0;
                const double x = t[o][side], y = g[o][side];
                if (kind == BC_COPY) field(f)[base + (side == 0 ? 1 : e - 2) * step] = x + y;
                else if (kind == BC_NEG || kind == BC_LIN2M) field(f)[base + (side == 0 ? 1 : e - 2) * step] = x - y;  // (homogeneous form)
            }
        return;
    }
    // BC_STRESS on the x2 / x3 faces (div_ghost, D = 1, 2): linear in V1 at the cell's two x1 faces, the other
    // tangential component and the normal one inside.  Alone in its stage.
    if (D == 0 || !on(D)) return;
    double* A = field(D);
#pragma unroll
    for (int side = 1; side >= 0; --side) {
        const int e = ext(D, D), cb = base + (side == 0 ? 0 : e - 1) * step, ci = base + (side == 0 ? 1 : e - 2) * step;
        const double g = A[cb];
        A[cb] = 0.0;
        if (g == 0.0) continue;
        const int cell = side == 0 ? 0 : e - 2, cc = base + cell * step;
        const int i = u, j = D == 1 ? cell : v;
        const CellMetric<double> m = cell_metric<double, G>(p, i, j);
        const double sgn = side == 0 ? -1.0 : 1.0, hc1 = 0.5 * m.c1, hc2 = 0.5 * m.c2;
        const double s = -g / (D == 1 ? fma(sgn, m.a2, hc2) : sgn * m.a3);
        atomicAdd(a.aV1 + cc, s * (hc1 - p.d1));
        atomicAdd(a.aV1 + cc + 1, s * (hc1 + p.d1));
        if (D == 1) {
            atomicAdd(a.aV3 + cc, -s * m.a3);
            atomicAdd(a.aV3 + cc + sz, s * m.a3);
            atomicAdd(A + ci, s * (hc2 - sgn * m.a2));
        } else {
            atomicAdd(a.aV2 + cc, s * (hc2 - m.a2));
            atomicAdd(a.aV2 + cc + sy, s * (hc2 + m.a2));
            atomicAdd(A + ci, -s * sgn * m.a3);
        }
    }
}

// pseudo-steps of the current viscosity (k_cells' DT_R) for the adjoint iteration
__global__ void __launch_bounds__(256) k_pt_dtr(KP<double> p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    const Dims& d = p.d;
    if (i >= d.n1 || j >= d.n2 || k >= d.n3) return;
    const int c = i + d.sy * j + d.sz * k;
    const double sm = p.etaSM[c], e = p.eta[c];
    const double gs = p.gsc * sm, kb = p.kbc * sm;
    p.DT_R[c] = p.vpdt2 / (kb + gs * (e / (e + gs)));
}

// λ_V of the transposed PT: λ_V += avg(DT_R) (Eᵀ μ + Dᵀ λ_P - b_V) at interior nodes
__global__ void __launch_bounds__(256) k_adj_velocity_update(const __grid_constant__ KP<double> p, const __grid_constant__ Adj a, double* lV1, double* lV2, double* lV3,
                                                             const double* bV1, const double* bV2, const double* bV3) {
    pdl_enter_small();
    const int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y * blockDim.y + threadIdx.y + 1, k = blockIdx.z + 1;
    const Dims& d = p.d;
    if (i > d.n1 - 1 || j > d.n2 - 1 || k > d.n3 - 1) return;
    const int sy = d.sy, sz = d.sz;
    const int c = i + sy * j + sz * k;
    const double h = 0.5;
    if (j <= d.n2 - 2 && k <= d.n3 - 2) lV1[c] += (a.aV1[c] - bV1[c]) * ((p.DT_R[c - 1] + p.DT_R[c]) * h);
    if (i <= d.n1 - 2 && k <= d.n3 - 2) lV2[c] += (a.aV2[c] - bV2[c]) * ((p.DT_R[c - sy] + p.DT_R[c]) * h);
    if (i <= d.n1 - 2 && j <= d.n2 - 2) lV3[c] += (a.aV3[c] - bV3[c]) * ((p.DT_R[c - sz] + p.DT_R[c]) * h);
}

// residual of the transposed system, r = Aᵀλ - b, in place of Aᵀλ (convergence check)
__global__ void __launch_bounds__(256) k_adj_residual(KP<double> p, Adj a, const double* bV1, const double* bV2, const double* bV3, const double* bP) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    const Dims& d = p.d;
    if (i > d.n1 || j > d.n2 || k > d.n3) return;
    const int sy = d.sy, sz = d.sz;
    const int c = i + sy * j + sz * k;
    const bool in1 = i >= 1 && i <= d.n1 - 1, in2 = j >= 1 && j <= d.n2 - 1, in3 = k >= 1 && k <= d.n3 - 1;
    a.aV1[c] = (in1 && in2 && in3 && j <= d.n2 - 2 && k <= d.n3 - 2) ? a.aV1[c] - bV1[c] : 0.0;
    a.aV2[c] = (in1 && in2 && in3 && i <= d.n1 - 2 && k <= d.n3 - 2) ? a.aV2[c] - bV2[c] : 0.0;
    a.aV3[c] = (in1 && in2 && in3 && i <= d.n1 - 2 && j <= d.n2 - 2) ? a.aV3[c] - bV3[c] : 0.0;
    a.aP[c] = (i < d.n1 && j < d.n2 && k < d.n3) ? a.aP[c] - bP[c] : 0.0;
}

}  // namespace sph
