// PT kernels that march along x3: one thread per (x1, x2) column, a chunk of planes each.
//
//   k_cells     compute_P! (WHAT_STRESS), with the strain rates kept for the strain-rate law
//               (WHAT_STRESS_LAW), the strain rates alone (WHAT_STRAIN) or the viscous stresses
//               and the divergence of the FP64 residual (WHAT_VISC)
//   k_nodes     compute_V!: V += avg(DT_R) (momentum) (MODE 0), with the right-hand side of the
//               correction problem (MODE 1), or the momentum residual itself (MODE 2)
//   k_edot      strain-rate power law; k_rheo compute_TII! + copy_BC!(τII) + power_law!
// (SphericalStokes_diapir.jl:155-329)
//
// Bound: FP64 instructions (sph_math.cuh).  A thread keeps its (x1, x2) position over the planes, so the
// metric factors are multiplied out with the spacings once per column (the kernels spent a third of
// their FP64 instructions on that per point), and the sums of η and ηSM over two cells of a plane serve the
// edges below and above it.  Columns are numbered along x1 over the whole plane, so that a
// ragged n1 leaves no idle lanes (an idle lane costs as much FP64 time as a busy one).  Loads are
// direct: neighbours come from L1, and their issue slots are free beside FP64 at 1/16 of a warp
// instruction per clock.
// Measured on a GB300, 127^3 sector, strain-rate law, us (FP64 operations per cell): k_cells with the strain
// rates kept 385 (98), k_nodes_law 352 (93), both with the FP64 units 87 % busy (spherical 63^3 73 and 84 %); one point per
// thread, with separate strain-rate kernel and CUDA's pow, exp and log: compute_P! 537, strain rates 223, law 642,
// compute_V! 310.  An iteration 765 (2071); Cartesian 207^3, relaxed stress law 3118 (7030).
#pragma once
#include "sph_math.cuh"

namespace sph {

// Threads per block.  No block shares anything, and the FP64 units of the fullest SM end last: single warps spread
// most evenly.  us per iteration with blocks of 128 and of 32: 63^3 116.9 and 114.1, sector 21 x 15 x 138 44.3 and
// 40.3, sector 110 x 28 x 30 64.1 and 60.2, 207^3 Cartesian 3372 and 3347, 127^3 sector 819 and 821.
constexpr int MC_NT = 32;

// planes per thread: enough to pay for the column's coefficients (`setup`, in planes), few enough for an even
// share of blocks per SM (the FP64 units are the only bound, so the fullest SM ends last) and for `need`
// times four warps per SM, below which the loads of a plane are not hidden behind its FP64 instructions; one more for
// the tail, where the last warps of an SM run alone
inline int march_chunk(long long columns, int planes, int sms, double setup, double need) {
    const long long cols = (columns + MC_NT - 1) / MC_NT;
    int best = 1;
    double best_t = 1e300;
    for (int k = 1; k <= 16 && k <= planes; ++k) {
        const long long blocks = cols * ((planes + k - 1) / k);
        const double n = (double)((blocks + sms - 1) / sms);
        const double t = ((n > 4 * need ? n : 4 * need) + 1.0) * (k + setup);
        if (t < best_t) { best_t = t; best = k; }
    }
    return best;
}

enum CellsWhat { WHAT_STRESS = 0, WHAT_STRESS_LAW, WHAT_STRAIN, WHAT_VISC };
// Resident blocks per SM that the registers of k_cells leave room for.  us a launch without a bound (123 registers) and with 20 (96):
// spherical 63^3, WHAT_STRESS, whose blocks are all resident at 20 only, 56.1 and 55.2; 127^3 sector, WHAT_STRESS_LAW,
// 384 and 385.
constexpr int cells_blocks(int what) { return what == WHAT_STRESS || what == WHAT_STRESS_LAW ? 20 : 24; }

// RHS: continuity right-hand side rP (P -= KBDT (div V + rP))
template <typename T, int G, int WHAT, bool RHS>
__global__ void __launch_bounds__(MC_NT, cells_blocks(WHAT)) k_cells(const __grid_constant__ KP<T> p, int chunk) {
    constexpr bool PT = WHAT == WHAT_STRESS || WHAT == WHAT_STRESS_LAW;
    constexpr bool ETA = WHAT != WHAT_STRAIN;
    pdl_enter_small();
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x;
    const int i = col % d.n1, j = col / d.n1;
    if (j >= d.n2) return;
    const int sy = d.sy, sz = d.sz;
    const int k0 = blockIdx.y * chunk, k1 = min(k0 + chunk, d.n3);
    const T h = T(0.5);
    // coefficients of the column: strain rates of the cell (sums of face velocities: halves folded in) and of its edges
    const CellMetric<T> m = cell_metric<T, G>(p, i, j);
    const EdgeMetric<T> e = edge_metric<T, G>(p.geo, i, j, d.n1, d.n2);
    const T a2 = m.a2, a3 = m.a3, e1 = h * m.e1, e2 = h * m.e2, third = T(-1.0 / 3.0);
    // (a difference and the sum of the same two values, d Δ + h (v + v'), as (d + h) Δ + 2 h v: one operation less)
    const T e12_2 = e.iRh * p.d2, e1_d = G != CART ? p.d1 - h * e.iRh : p.d1, e1_v = -e.iRh;
    const T e13_3 = G == SPH ? e.iRh * e.iSc1 * p.d3 : p.d3, e13_d = G == SPH ? e1_d : p.d1;
    const T e23_2 = G == SPH ? e.iRc1 * p.d2 - h * e.iRc1 * e.ctH : e.iRc1 * p.d2, e23_v = -e.iRc1 * e.ctH;
    const T e23_3 = G == SPH ? e.iRc1 * e.iSh * p.d3 : p.d3;
    const bool v12 = i < d.n1 - 1 && j < d.n2 - 1, v13 = i < d.n1 - 1 && j < d.n2 - 2, v23 = i < d.n1 - 2 && j < d.n2 - 1;
    int c = i + sy * j + sz * k0;
    // Sums over two cells of a plane: X along x1 in row j + 1, Y along x2 in column i + 1.  Cells past the grid are
    // replaced by the last ones inside (their edges are not stored), so that `mid` tells of cells of the grid only.
    const int ox = i < d.n1 - 1 ? 1 : 0, oy = j < d.n2 - 1 ? sy : 0;
    T eX = T(0), eY = T(0), sX = T(0), sY = T(0);
    // whether the quotients of this column may be formed by mid_div: its steps, and η and ηSM of the plane below
    bool steps = true, below = true;
    if (PT) {
        MidRange<T, 100> m;
        m.add(p.gsc); m.add(p.kbc); m.add(p.vpdt2);
        steps = m.ok();
    }
    {
        MidRange<T, 400> m;
        if (ETA) {
            const T a = p.eta[c + ox], b = p.eta[c + oy], q = p.eta[c + ox + oy];
            eX = b + q; eY = a + q;
            if (PT) { m.add(p.eta[c]); m.add(a); m.add(b); m.add(q); }
        }
        if (PT) {
            const T a = p.etaSM[c + ox], b = p.etaSM[c + oy], q = p.etaSM[c + ox + oy];
            sX = b + q; sY = a + q;
            m.add(p.etaSM[c]); m.add(a); m.add(b); m.add(q);
            below = steps && m.ok();
        }
    }
    const T gsc4 = T(0.25) * p.gsc;
    // (velocities past the grid are padding of the box: finite, and their results are not stored)
    for (int k = k0; k < k1; ++k, c += sz) {
        const int u = c + sz;
        // sums of the plane above; edges of it: sums e, s of η and ηSM over four cells
        T e12 = T(0), e13 = T(0), e23 = T(0), s12 = T(0), s13 = T(0), s23 = T(0);
        const int w = k < d.n3 - 1 ? u : c;
        MidRange<T, 400> mid;
        if (ETA) {
            const T o = p.eta[w], a = p.eta[w + ox], b = p.eta[w + oy], q = p.eta[w + ox + oy];
            const T x = b + q, y = a + q;
            e12 = (o + a) + x; e13 = eX + x; e23 = eY + y;
            eX = x; eY = y;
            if (PT) { mid.add(o); mid.add(a); mid.add(b); mid.add(q); }
        }
        if (PT) {
            const T o = p.etaSM[w], a = p.etaSM[w + ox], b = p.etaSM[w + oy], q = p.etaSM[w + ox + oy];
            const T x = b + q, y = a + q;
            s12 = gsc4 * ((o + a) + x); s13 = gsc4 * (sX + x); s23 = gsc4 * (sY + y);  // aG = GSDT s / 4
            sX = x; sY = y;
            mid.add(o); mid.add(a); mid.add(b); mid.add(q);
        }
        const T v1p = p.V1[c + 1], v2p = p.V2[c + sy], v3p = p.V3[u];
        const T D1 = v1p - p.V1[c], D2 = v2p - p.V2[c], D3 = v3p - p.V3[c];
        T D11 = p.d1 * D1, D22, D33, div;
        if (G != CART) {
            const T ex = e1 * (p.V1[c] + v1p);
            D22 = fma(a2, D2, ex);
            D33 = G == SPH ? fma(a3, D3, fma(e2, p.V2[c] + v2p, ex)) : a3 * D3;
            div = D11 + D22 + D33;
            D11 = fma(div, third, D11); D22 = fma(div, third, D22); D33 = fma(div, third, D33);
        } else {
            D22 = a2 * D2; D33 = a3 * D3;
            div = D11 + D22 + D33;
        }
        const T v1a = p.V1[u + 1], v1b = p.V1[u + 1 + sy], v2a = p.V2[u + sy], v2b = p.V2[u + sy + 1];
        const T v3q = p.V3[u + sy], v3t = p.V3[u + sy + 1], v3s = p.V3[u + 1];
        T D12 = fma(e12_2, v1b - v1a, e1_d * (v2b - v2a));
        if (G != CART) D12 = fma(e1_v, v2a, D12);
        T D13 = fma(e13_3, v1b - p.V1[c + 1 + sy], e13_d * (v3t - v3q));
        if (G == SPH) D13 = fma(e1_v, v3q, D13);
        T D23 = fma(e23_3, v2b - p.V2[c + 1 + sy], e23_2 * (v3t - v3s));
        if (G == SPH) D23 = fma(e23_v, v3s, D23);
        const bool w12 = v12 && k < d.n3 - 2, w13 = v13 && k < d.n3 - 1, w23 = v23 && k < d.n3 - 1;
        if (WHAT == WHAT_STRAIN || WHAT == WHAT_STRESS_LAW) {
            p.sDD[c] = h * fma(D11, D11, fma(D22, D22, D33 * D33));
            if (w12) p.s12[c] = D12;
            if (w13) p.s13[c] = D13;
            if (w23) p.s23[c] = D23;
        }
        if (PT) {
            const T et = p.eta[c], sm = p.etaSM[c];
            const T gs = p.gsc * sm, kb = p.kbc * sm, gs2 = gs + gs;
            const T m11 = fma(gs2, D11, p.t11[c]), m22 = fma(gs2, D22, p.t22[c]), m33 = fma(gs2, D33, p.t33[c]);
            const T m12 = fma(s12, D12, p.t12[c]), m13 = fma(s13, D13, p.t13[c]), m23 = fma(s23, D23, p.t23[c]);
            T Pn = fma(-kb, RHS ? div + p.rP[c] : div, p.P[c]);
            // 1/(1 + GSDT/η), the step, and at the edges aE / (aE + aG), aE = e / 4.  One rare branch for all five,
            // behind the loads of the plane: a branch for each cost 10 % of an iteration, one before the loads 4 %.
            const T b0 = et + gs, b12 = fma(T(4), s12, e12), b13 = fma(T(4), s13, e13), b23 = fma(T(4), s23, e23);
            T f = mid_div(et, b0), dt = mid_div(p.vpdt2, fma(gs, f, kb)), q12 = mid_div(e12, b12), q13 = mid_div(e13, b13), q23 = mid_div(e23, b23);
            const bool above = steps && mid.ok();
            if (__builtin_expect(!(below && above), 0)) {
                f = et / b0;
                dt = p.vpdt2 / fma(gs, f, kb);
                q12 = e12 / b12; q13 = e13 / b13; q23 = e23 / b23;
            }
            below = above;
            const T n11 = m11 * f, n22 = m22 * f, n33 = m33 * f;
            if (p.traction) traction_pressure(j, k, d.n2, d.n3, n22, n33, p.sig2, p.sig3, Pn);
            if (p.fs && i == d.n1 - 1) Pn = fs_pressure(n11, p.top_load ? p.top_load[c] : T(0), p.fs_kappa, p.V1[c], v1p);
            p.P[c] = Pn;
            p.t11[c] = n11; p.t22[c] = n22; p.t33[c] = n33;
            p.DT_R[c] = dt;
            if (w12) p.t12[c] = m12 * q12;
            if (w13) p.t13[c] = m13 * q13;
            if (w23) p.t23[c] = m23 * q23;
        } else if (WHAT == WHAT_VISC) {
            const T x = T(2) * p.eta[c];
            p.t11[c] = x * D11; p.t22[c] = x * D22; p.t33[c] = x * D33;
            p.rP[c] = div;
            if (w12) p.t12[c] = T(0.25) * e12 * D12;
            if (w13) p.t13[c] = T(0.25) * e13 * D13;
            if (w23) p.t23[c] = T(0.25) * e23 * D23;
        }
    }
}

template <typename T, int G, int MODE>
__device__ __forceinline__ void nodes_body(const KP<T>& p, int chunk, int by) {
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x;
    const int w = d.n1 - 1;
    const int I = col % w + 1, J = col / w + 1;
    if (J > d.n2 - 1) return;
    const int sy = d.sy, sz = d.sz;
    const int K0 = by * chunk + 1, K1 = min(K0 + chunk, d.n3);  // K0 .. K1 - 1
    // the update wants the residual times (DT + DT') / 2: its half is folded into the coefficients
    const T s = MODE == 2 ? T(1) : T(0.5), h = T(0.5);
    const MomMetric<T> m = mom_metric<T, G>(p.geo, I, J, d.n1, d.n2);
    // coefficients of differences, and of the lower value where its sum with the upper one enters too:
    // d Δ + h (v + v') = (d + h) Δ + 2 h v
    const T c1 = s * p.d1;
    const T m1_n = s * (G == SPH ? m.iR1 : h * m.iR1), m1_t = G == SPH ? s * h * m.iR1 * m.ct1 : T(0);
    const T m1_1 = G == CART ? c1 : c1 + m1_n, m1_2 = s * m.iR1 * p.d2 + m1_t, m1_3 = s * (G == SPH ? m.iR1 * m.iS1 * p.d3 : p.d3);
    const T m2_s = G == CART ? T(0) : s * (G == SPH ? T(1.5) * m.iR2 : m.iR2), m2_n = G == SPH ? s * h * m.iR2 * m.ct2 : T(0);
    const T m2_1 = c1 + m2_s, m2_2 = s * m.iR2 * p.d2 + m2_n, m2_3 = s * (G == SPH ? m.iR2 * m.iS2 * p.d3 : p.d3);
    const T m3_s = G == CART ? T(0) : s * (G == SPH ? T(1.5) * m.iR2 : h * m.iR2), m3_n = G == SPH ? s * m.iR2 * m.ct3 : T(0);
    const T m3_1 = c1 + m3_s, m3_2 = s * m.iR2 * p.d2 + m3_n, m3_3 = s * (G == SPH ? m.iR2 * m.iS3 * p.d3 : p.d3);
    const T gh = -s * h * p.g;
    const bool w1 = J <= d.n2 - 2, w2 = I <= d.n1 - 2, w3 = w1 && w2;
    int c = I + sy * J + sz * K0;
    // plane K0 - 1: σ33 and DT_R of the cell below, edge stresses
    T q33 = p.t33[c - sz] - p.P[c - sz], qdt = MODE == 2 ? T(0) : p.DT_R[c - sz];
    T p13a = p.t13[c - sy - sz], p13b = p.t13[c - 1 - sy - sz], p23 = p.t23[c - 1 - sy - sz];
    for (int K = K0; K < K1; ++K, c += sz) {
        const T P = p.P[c];
        const T s11 = p.t11[c] - P, s22 = p.t22[c] - P, s33 = p.t33[c] - P;
        const T dt = MODE == 2 ? T(0) : p.DT_R[c];
        const T t13a = p.t13[c - sy], t13b = p.t13[c - 1 - sy], t23 = p.t23[c - 1 - sy];
        const T t12b = p.t12[c - 1 - sy - sz], t12c = p.t12[c - sy - sz];
        const bool kin = K <= d.n3 - 2;
        auto put = [&](T* V, T* R, T r, T dm) {
            if (MODE == 2) R[c] = r;
            else V[c] = fma(MODE == 1 ? fma(h, R[c], r) : r, dm + dt, V[c]);
        };
        if (w1 && kin) {  // V1 (I-1/2, J, K), cell m = (I-1, J, K)
            const T Pm = p.P[c - 1], t12a = p.t12[c - 1 - sz];
            const T m11 = p.t11[c - 1] - Pm;
            T r = fma(m1_3, t13b - p13b, fma(m1_2, t12a - t12b, m1_1 * (s11 - m11)));
            if (G == SPH) {
                const T m22 = p.t22[c - 1] - Pm, m33 = p.t33[c - 1] - Pm;
                r = fma(T(2) * m1_t, t12b, fma(m1_n, fma(-h, (m22 + s22) + (m33 + s33), m11 + m11), r));
            } else if (G == CYL) {
                r = fma(m1_n, (m11 + m11) - (p.t22[c - 1] - Pm + s22), r);
            }
            if (G != CART && MODE != 1) r = fma(gh, p.rho[c - 1] + p.rho[c], r);
            put(p.V1, p.rV1, r, MODE == 2 ? T(0) : p.DT_R[c - 1]);
        }
        if (w2 && kin) {  // V2 (I, J-1/2, K), cell m = (I, J-1, K)
            const T Pm = p.P[c - sy];
            const T m22 = p.t22[c - sy] - Pm;
            T r = fma(m2_3, t23 - p23, fma(m2_2, s22 - m22, m2_1 * (t12c - t12b)));
            if (G != CART) r = fma(T(2) * m2_s, t12b, r);
            if (G == SPH) r = fma(m2_n, (m22 + m22) - (p.t33[c - sy] - Pm + s33), r);
            put(p.V2, p.rV2, r, MODE == 2 ? T(0) : p.DT_R[c - sy]);
        }
        if (w3) {  // V3 (I, J, K-1/2), cell m = (I, J, K-1)
            const T t23a = p.t23[c - 1 - sz];
            T r = fma(m3_3, s33 - q33, fma(m3_2, t23a - p23, m3_1 * (p13a - p13b)));
            if (G != CART) r = fma(T(2) * m3_s, p13b, r);
            if (G == SPH) r = fma(T(2) * m3_n, p23, r);
            if (G == CART && MODE != 1) r = fma(gh, p.rho[c - sz] + p.rho[c], r);
            put(p.V3, p.rV3, r, qdt);
        }
        q33 = s33; qdt = dt; p13a = t13a; p13b = t13b; p23 = t23;
    }
}
template <typename T, int G, int MODE>
__global__ void __launch_bounds__(MC_NT) k_nodes(const __grid_constant__ KP<T> p, int chunk) {
    pdl_enter_small();
    nodes_body<T, G, MODE>(p, chunk, blockIdx.y);
}

// strain-rate power law (k_edot_law of sph_pt.cuh is the FP32 one): with x = (ε̇_II / ε̇_bg)^2 of the clamped
// interior cell, η_t = 2 / (1/η_ini + 1/η_PL) = 2 η_ini / (1 + x^((n-1)/(2n))); RELAXED: η_out = η^(1-relax) η_t^relax
template <bool RELAXED>
__device__ __forceinline__ void edot_body(const KP<double>& p, int chunk, int by) {
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x;
    const int i = col % d.n1, j = col / d.n1;
    if (j >= d.n2) return;
    const int sy = d.sy, sz = d.sz;
    const int k0 = by * chunk, k1 = min(k0 + chunk, d.n3);
    const double* tab = p.geo.pow_tab;
    const int s0 = clampi(i, 1, d.n1 - 2) + sy * clampi(j, 1, d.n2 - 2);
    int last = -1;
    double x = 0.0, b0 = 0.0, q0 = 0.0;  // the invariant squared; sums of the edges below the next plane
    for (int k = k0; k < k1; ++k) {
        const int kc = clampi(k, 1, d.n3 - 2);
        const int c = i + sy * j + sz * k;
        if (kc != last) {
            const int s = s0 + sz * kc, e = s - 1 - sy - sz;
            if (last < 0) { b0 = p.s13[e] + p.s13[e + 1]; q0 = p.s23[e] + p.s23[e + sy]; }
            const double a = (p.s12[e] + p.s12[e + sy]) + (p.s12[e + 1] + p.s12[e + 1 + sy]);
            const double b1 = p.s13[e + sz] + p.s13[e + 1 + sz], q1 = p.s23[e + sz] + p.s23[e + sy + sz];
            const double b = b0 + b1, q = q0 + q1;
            b0 = b1; q0 = q1;
            // (sums of four edges: a quarter of each, squared, times another quarter)
            x = fma(1.0 / 64.0, fma(a, a, fma(b, b, q * q)), p.sDD[s]);
            last = kc;
        }
        const double ei = p.eta_ini[c], eo = RELAXED ? p.eta[c] : ei, w = x * p.law_i2;
        const bool lin = p.phase && p.phase[c], half = p.relax == 0.5;
        double et = ei;
        const bool rest = __double_as_longlong(x) == 0, root = root_range(w);
        MidRange<double, 400> mid;
        mid.add(ei); mid.add(eo);
        if (p.law_q && (half || !RELAXED) && mid.ok() && (root || rest)) {  // (every intermediate value is a normal number, or zero)
            double f = 0.0;
            if (root) f = root_pow(w, p.law_p, p.law_q, p.law_rho, p.law_e, p.law_el);
            if (!lin) et = mid_div(ei + ei, 1.0 + f);
            if (RELAXED) et = mid_sqrt(eo * et);
        } else {
            if (!lin) {
                double f;
                if (p.law_q && root) f = root_pow(w, p.law_p, p.law_q, p.law_rho, p.law_e, p.law_el);
                else if (normal_pos(w)) f = fast_pow(tab, w, p.law_ex);
                else if (rest && p.law_ex > 0.0) f = 0.0;
                else f = pow(sqrt(x) / p.edot_bg, 2.0 * p.law_ex);  // (the square of the ratio leaves the range first)
                et = near_div(ei + ei, 1.0 + f);
            }
            if (RELAXED) {
                // the half-way mean as a root, else η (η_t/η)^relax; by logarithms where the product or the quotient is no
                // normal number (a cell without viscosity keeps none)
                const double r = half ? eo * et : near_div(et, eo);
                if (normal_pos(r)) et = half ? fast_sqrt(r) : eo * fast_pow(tab, r, p.relax);
                else et = exp((1.0 - p.relax) * log(eo) + p.relax * log(et));
            }
        }
        p.eta_out[c] = et;
    }
}
template <bool RELAXED>
__global__ void __launch_bounds__(MC_NT) k_edot(const __grid_constant__ KP<double> p, int chunk) {
    pdl_enter_small();
    edot_body<RELAXED>(p, chunk, blockIdx.y);
}

// compute_TII! + copy_BC!(τII) + power_law! (k_rheo_tau of sph_pt.cuh is the FP32 one): with x = (τII / τ_C)^2,
// η_PL = η_ini x^((1-n)/2), η = 2 / (1/η_ini + 1/η_PL); RELAX: η_PL relaxed in log space
// (CylindricalStokes_diapir.jl:185-192).  phase == 1 cells are linear.
template <bool RELAX>
__device__ __forceinline__ void rheo_body(const KP<double>& p, int faces_only, int chunk, int by) {
    const Dims& d = p.d;
    const int col = blockIdx.x * MC_NT + threadIdx.x;
    const int i = col % d.n1, j = col / d.n1;
    if (j >= d.n2) return;
    const int sy = d.sy, sz = d.sz;
    const int k0 = by * chunk, k1 = min(k0 + chunk, d.n3);
    const double* tab = p.geo.pow_tab;
    const int s0 = clampi(i, 1, d.n1 - 2) + sy * clampi(j, 1, d.n2 - 2);
    const int rim = (i == 0 || i == d.n1 - 1) + (j == 0 || j == d.n2 - 1);
    int last = -1;
    double t2c = 0.0, tiic = 0.0, b0 = 0.0, q0 = 0.0;
    for (int k = k0; k < k1; ++k) {
        const int c = i + sy * j + sz * k;
        double t2, tii;
        if (faces_only && rim + (k == 0 || k == d.n3 - 1) >= 2) {
            tii = p.tII[c];  // CartesianStokes_diapir.jl:97-105 never writes edges/corners of τII
            t2 = tii * tii;
        } else {
            const int kc = clampi(k, 1, d.n3 - 2);
            if (kc != last) {
                const int s = s0 + sz * kc, e = s - 1 - sy - sz;
                if (last < 0) { b0 = p.t13[e] + p.t13[e + 1]; q0 = p.t23[e] + p.t23[e + sy]; }
                const double a = (p.t12[e] + p.t12[e + sy]) + (p.t12[e + 1] + p.t12[e + 1 + sy]);
                const double b1 = p.t13[e + sz] + p.t13[e + 1 + sz], q1 = p.t23[e + sz] + p.t23[e + sy + sz];
                const double b = b0 + b1, q = q0 + q1;
                b0 = b1; q0 = q1;
                const double x = p.t11[s], y = p.t22[s], z = p.t33[s];
                t2c = fma(0.5, fma(x, x, fma(y, y, z * z)), 1.0 / 16.0 * fma(a, a, fma(b, b, q * q)));
                tiic = fast_sqrt(t2c);
                last = kc;
            }
            t2 = t2c;
            p.tII[c] = tii = tiic;
        }
        const bool lin = p.phase && p.phase[c];
        const double cx = lin ? 0.0 : p.law_ex;
        const double ei = p.eta_ini[c], x = t2 * p.law_i2;
        // integer n: (τII / τ_C)^(n-1) by multiplication
        const double w = p.law_q ? small_pow(tii * p.law_i1, x, lin ? 0 : p.law_p) : 0.0;
        if (!RELAX) {
            double f = w;
            if (!p.law_q) {  // (as in edot_body)
                if (normal_pos(x)) f = fast_pow(tab, x, cx);
                else f = __double_as_longlong(t2) == 0 && cx > 0.0 ? 0.0 : pow(tii / p.tau_C, 2.0 * cx);
            }
            p.eta[c] = near_div(ei + ei, 1.0 + f);
        } else {
            const double po = p.eta_pl[c];
            double pl;
            bool done = false;
            if (p.law_q) {  // η_PL' = po (ei / (po w))^relax
                const double den = po * w;
                // (η_PL itself, ei / w, has to be a normal number too: where it is not, it is 0 or infinite, as in power_law!)
                const int ex = (__double2hiint(ei) >> 20) - (__double2hiint(w) >> 20);
                if (normal_pos(w) && normal_pos(ei) && normal_pos(po) && normal_pos(den) && ex > -1000 && ex < 1000) {
                    const double r = near_div(ei, den);
                    if (normal_pos(r)) {
                        double h, t;
                        log2_parts(tab, r, h, t);
                        const double y = p.relax * h;
                        if ((__double2hiint(y) & 0x7fffffff) < 0x408f4000) {  // |y| < 1000
                            pl = po * exp2_parts(tab, y, fma(p.relax, t, fma(p.relax, h, -y)));
                            done = true;
                        }
                    }
                }
            } else if (normal_pos(x) && normal_pos(ei) && normal_pos(po)) {
                // η_PL' = po 2^(relax (log2 ei - log2 po - cx log2 x)), the exponent as a head and a tail
                double hx, tx, hi, ti, ho, to;
                log2_parts(tab, x, hx, tx);
                log2_parts(tab, ei, hi, ti);
                log2_parts(tab, po, ho, to);
                const double L = hi - ho, q = cx * hx, s = L - q;
                const double low = ((ti - to) - fma(cx, tx, fma(cx, hx, -q))) + ((L - s) - q);
                const double y = p.relax * s;
                // |y| < 1000, and η_PL before the relaxation a normal number
                if ((__double2hiint(y) & 0x7fffffff) < 0x408f4000 && (__double2hiint(hi - q) & 0x7fffffff) < 0x408f4000) {
                    pl = po * exp2_parts(tab, y, fma(p.relax, low, fma(p.relax, s, -y)));
                    done = true;
                }
            }
            if (!done) {
                pl = ei * pow(tii / p.tau_C, -2.0 * cx);
                pl = exp(log(pl) * p.relax + log(po) * (1.0 - p.relax));
            }
            p.eta_pl[c] = pl;
            const double num = (ei + ei) * pl;
            p.eta[c] = done && normal_pos(num) ? near_div(num, ei + pl) : 2.0 / (1.0 / ei + 1.0 / pl);
        }
    }
}

template <bool RELAX>
__global__ void __launch_bounds__(MC_NT) k_rheo(const __grid_constant__ KP<double> p, int faces_only, int chunk) {
    pdl_enter_small();
    rheo_body<RELAX>(p, faces_only, chunk, blockIdx.y);
}

// compute_V! and the viscosity law of one iteration in one launch: both follow the stresses and neither reads what
// the other writes.  Blocks y < ny update the velocities, the others the viscosity.  LAW 0, 1: stress power law, plain
// and relaxed; 2: strain-rate power law, relaxed.  With ηSM of the next iteration in the boundary launch (k_bc), three
// launches an iteration in place of five; us per iteration: 70 x 5 x 5 18.6 and 12.9, spherical 63^3 114.0 and 107.7,
// 127^3 sector 818 and 797, sector 21 x 15 x 138 39.6 and 35.7, FP32 95 x 79 x 67 (four launches, three) 33.9 and 30.9.
template <int G, int LAW>
__global__ void __launch_bounds__(MC_NT) k_nodes_law(const __grid_constant__ KP<double> p, int faces_only, int kn, int ny, int kl) {
    pdl_enter_small();
    const int by = blockIdx.y;
    if (by < ny) nodes_body<double, G, 0>(p, kn, by);
    else if (LAW == 2) edot_body<true>(p, kl, by - ny);
    else rheo_body<LAW == 1>(p, faces_only, kl, by - ny);
}

}  // namespace sph
