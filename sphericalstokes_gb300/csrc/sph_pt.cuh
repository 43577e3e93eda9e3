// Pseudo-transient kernels (one thread per grid point, direct global access).
//
// These are the building blocks of one PT iteration in the reference's order
// (SphericalStokes_diapir.jl:413-425):
//   k_maxloc   maxloc! + copy_BC!(ηSM)          :149-152, :102-124
//   k_cells    compute_P!                        :155-241   (sph_march.cuh)
//   k_rheo_tau compute_TII! + copy_BC!(τII) + power_law!   :243-265 (FP64: k_rheo, sph_march.cuh)
//   k_edot_law strain-rate power law (not in the reference; FP64: k_edot, sph_march.cuh)
//   k_nodes    compute_V!                        :267-329   (sph_march.cuh)
//   k_bc       BC_R! / BC_θ! / BC_φ! and the cyl/cart BC kernels, all stages
// All three coordinate systems share the kernels; the metric terms come from
// the template parameter G and the 1D tables in Geo.  The FP32 fused sweeps in
// sph_sweep.cuh and sph_fused.cuh implement the same arithmetic with shared-memory tiling.
#pragma once
#include "sph_core.cuh"

namespace sph {

// ---------------------------------------------------------------------------
// ηSM = 7-point maximum of η on interior cells; boundary cells take the value
// of the clamped interior cell (copy_bc_r!, copy_bc_θ!, copy_bc_φ! in that
// order leave exactly that).  faces_only: CartesianStokes_diapir.jl:97-105
// copies only face interiors and edges/corners keep η (ηSM .= η before maxloc!).
//
// The maximum is taken on integers in the numbers' order (a comparison in FP64 would cost FP64
// issue, three of them per jmax): the bits of x with the magnitude of a negative x flipped, every
// NaN above +inf, so that it propagates as in Julia's maximum.
__device__ __forceinline__ long long order_bits(double x) {
    const long long b = __double_as_longlong(x);
    if ((b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL) return 0x7fffffffffffffffLL;
    return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double from_order(long long b, double) { return __longlong_as_double(b ^ ((b >> 63) & 0x7fffffffffffffffLL)); }
__device__ __forceinline__ int order_bits(float x) {
    const int b = __float_as_int(x);
    if ((b & 0x7fffffff) > 0x7f800000) return 0x7fffffff;
    return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float from_order(int b, float) { return __int_as_float(b ^ ((b >> 31) & 0x7fffffff)); }
template <typename T>
__device__ __forceinline__ void maxloc_body(const KP<T>& p, int faces_only, int i, int j, int k) {
    const Dims& d = p.d;
    if (i >= d.n1 || j >= d.n2 || k >= d.n3) return;
    const int c = i + d.sy * j + d.sz * k;
    int nb = (i == 0 || i == d.n1 - 1) + (j == 0 || j == d.n2 - 1) + (k == 0 || k == d.n3 - 1);
    if (faces_only && nb >= 2) { p.etaSM[c] = p.eta[c]; return; }
    const int a = clampi(i, 1, d.n1 - 2), b = clampi(j, 1, d.n2 - 2), e = clampi(k, 1, d.n3 - 2);
    const int s = a + d.sy * b + d.sz * e;
    const T* E = p.eta;
    auto m = order_bits(E[s]);
    const int off[6] = {-1, 1, -d.sy, d.sy, -d.sz, d.sz};
    for (int q = 0; q < 6; ++q) m = max(m, order_bits(E[s + off[q]]));
    p.etaSM[c] = from_order(m, T(0));
}
template <typename T>
__global__ void k_maxloc(const __grid_constant__ KP<T> p, int faces_only) {
    pdl_enter_small();
    maxloc_body(p, faces_only, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.y * blockDim.y + threadIdx.y, blockIdx.z);
}

// ---------------------------------------------------------------------------
// strain rates of the current velocities as separate fields (the DIVV and D_*
// arrays compute_P! fills in CylindricalStokes_diapir.jl:153-159): divergence
// and normal rates at cells, engineering shear rates at the three edge sets,
// in the layout of P and τ12, τ13, τ23.
template <typename T, int G>
__global__ void __launch_bounds__(256) k_strain_out(KP<T> p, T* __restrict__ dv, T* __restrict__ d11, T* __restrict__ d22,
                                                    T* __restrict__ d33, T* __restrict__ d12, T* __restrict__ d13, T* __restrict__ d23) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    const Dims& d = p.d;
    if (i >= d.n1 || j >= d.n2 || k >= d.n3) return;
    const int sy = d.sy, sz = d.sz;
    const int c = i + sy * j + sz * k;
    const CellD<T> D = cell_strain<T, G>(p.geo, p.d1, p.d2, p.d3, i, j, p.V1[c], p.V1[c + 1], p.V2[c], p.V2[c + sy], p.V3[c], p.V3[c + sz]);
    dv[c] = D.div; d11[c] = D.D11; d22[c] = D.D22; d33[c] = D.D33;
    if (i < d.n1 - 1 && j < d.n2 - 1 && k < d.n3 - 2) {
        const int q = c + sz;
        d12[c] = edge12<T, G>(p.geo, p.d1, p.d2, i, p.V2[q + sy], p.V2[q + sy + 1], p.V1[q + 1], p.V1[q + 1 + sy]);
    }
    if (i < d.n1 - 1 && j < d.n2 - 2 && k < d.n3 - 1) {
        const int q = c + sy;
        d13[c] = edge13<T, G>(p.geo, p.d1, p.d3, i, j, p.V3[q + sz], p.V3[q + sz + 1], p.V1[q + 1], p.V1[q + 1 + sz]);
    }
    if (i < d.n1 - 2 && j < d.n2 - 1 && k < d.n3 - 1) {
        const int q = c + 1;
        d23[c] = edge23<T, G>(p.geo, p.d2, p.d3, i, j, p.V3[q + sz], p.V3[q + sz + sy], p.V2[q + sy], p.V2[q + sy + sz]);
    }
}

// ---------------------------------------------------------------------------
// second invariant of τ at an interior cell s (compute_TII!, :246-255)
template <typename T>
__device__ __forceinline__ T tau_II(const KP<T>& p, int s) {
    const int sy = p.d.sy, sz = p.d.sz;
    const T q4 = T(0.25);
    const int e = s - 1 - sy - sz;  // edge (I-1, J-1, K-1)
    const T a = (p.t12[e] + p.t12[e + sy] + p.t12[e + 1] + p.t12[e + 1 + sy]) * q4;
    const T b = (p.t13[e] + p.t13[e + sz] + p.t13[e + 1] + p.t13[e + 1 + sz]) * q4;
    const T c = (p.t23[e] + p.t23[e + sz] + p.t23[e + sy] + p.t23[e + sy + sz]) * q4;
    const T x = p.t11[s], y = p.t22[s], z = p.t33[s];
    return sqrt(T(0.5) * (x * x + y * y + z * z) + a * a + b * b + c * c);
}

// compute_TII! + copy_BC!(τII) + power_law! (RELAX: log-space relaxation of
// η_PL, CylindricalStokes_diapir.jl:185-192).  phase==1 cells are linear.
// Its launch overlaps the end of the sweep before it: FP32 iteration at 95 x 79 x 67 30.9 us without, 29.2 with.
template <typename T, bool RELAX>
__global__ void k_rheo_tau(KP<T> p, int faces_only, T n_exp) {
    pdl_enter_small();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    const Dims& d = p.d;
    if (i >= d.n1 || j >= d.n2 || k >= d.n3) return;
    const int c = i + d.sy * j + d.sz * k;
    const int nb = (i == 0 || i == d.n1 - 1) + (j == 0 || j == d.n2 - 1) + (k == 0 || k == d.n3 - 1);
    T tii;
    if (faces_only && nb >= 2) {
        tii = p.tII[c];  // CartesianStokes_diapir.jl:97-105 never writes edges/corners of τII
    } else {
        const int s = clampi(i, 1, d.n1 - 2) + d.sy * clampi(j, 1, d.n2 - 2) + d.sz * clampi(k, 1, d.n3 - 2);
        tii = tau_II(p, s);
        p.tII[c] = tii;
    }
    const T ne = (p.phase && p.phase[c]) ? T(1) : n_exp;
    const T ei = p.eta_ini[c];
    if (!RELAX) {
        p.eta[c] = T(2) / (T(1) / ei + T(1) / (ei * pow(tii / p.tau_C, T(1) - ne)));
    } else {
        T pl = ei * pow(tii / p.tau_C, T(1) - ne);
        pl = exp(log(pl) * p.relax + log(p.eta_pl[c]) * (T(1) - p.relax));
        p.eta_pl[c] = pl;
        p.eta[c] = T(2) / (T(1) / ei + T(1) / pl);
    }
}

// strain-rate power law (not in the reference): the invariant of the clamped
// interior cell (as copy_BC! does for τII), η_t = 2/(1/η_ini + 1/η_PL),
// η_PL = η_ini (edot_II/edot_bg)^((1-n)/n); RELAXED: η_out = η^(1-relax) η_t^relax.
template <typename T, bool RELAXED>
__global__ void k_edot_law(KP<T> p) {
    pdl_enter_small();
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    const Dims& d = p.d;
    if (i >= d.n1 || j >= d.n2 || k >= d.n3) return;
    const int sy = d.sy, sz = d.sz;
    const int c = i + sy * j + sz * k;
    const int s = clampi(i, 1, d.n1 - 2) + sy * clampi(j, 1, d.n2 - 2) + sz * clampi(k, 1, d.n3 - 2);
    const T q4 = T(0.25);
    const int e = s - 1 - sy - sz;
    const T a = (p.s12[e] + p.s12[e + sy] + p.s12[e + 1] + p.s12[e + 1 + sy]) * q4;
    const T b = (p.s13[e] + p.s13[e + sz] + p.s13[e + 1] + p.s13[e + 1 + sz]) * q4;
    const T cc = (p.s23[e] + p.s23[e + sz] + p.s23[e + sy] + p.s23[e + sy + sz]) * q4;
    const T ed = sqrt(p.sDD[s] + q4 * (a * a + b * b + cc * cc));
    const T ei = p.eta_ini[c];
    T et;
    if (p.phase && p.phase[c]) {
        et = ei;
    } else {
        const T pl = ei * pow(ed / p.edot_bg, (T(1) - p.n_exp) / p.n_exp);
        et = T(2) / (T(1) / ei + T(1) / pl);
    }
    p.eta_out[c] = RELAXED ? exp((T(1) - p.relax) * log(p.eta[c]) + p.relax * log(et)) : et;
}

// ---------------------------------------------------------------------------
// compute_V!: momentum residuals at interior velocity nodes (:267-307).
// GRAV: include the ρg body force; RHS: add the right-hand side rV instead.
// ok[f] tells whether (I,J,K) is an interior node of velocity component f.
template <typename T, int G, bool GRAV, bool RHS>
__device__ __forceinline__ void momentum(const KP<T>& p, int I, int J, int K, T dv[3], bool ok[3]) {
    const Dims& d = p.d;
    const int sy = d.sy, sz = d.sz;
    const int c = I + sy * J + sz * K;
    const T h = T(0.5);
    const T Pc = p.P[c];
    const T s11 = p.t11[c] - Pc, s22 = p.t22[c] - Pc, s33 = p.t33[c] - Pc;
    ok[0] = (J <= d.n2 - 2 && K <= d.n3 - 2);
    ok[1] = (I <= d.n1 - 2 && K <= d.n3 - 2);
    ok[2] = (I <= d.n1 - 2 && J <= d.n2 - 2);
    if (ok[0]) {  // V1 (I-1/2, J, K)
        const int m = c - 1;
        const T Pm = p.P[m];
        T r = mom1<T, G>(p.geo, p.d1, p.d2, p.d3, I, J, p.t11[m] - Pm, s11, p.t22[m] - Pm, s22, p.t33[m] - Pm, s33,
                         p.t12[m - sz], p.t12[m - sy - sz], p.t13[m - sy], p.t13[m - sy - sz]);
        if (G != CART && GRAV) r -= (p.rho[m] * p.g + p.rho[c] * p.g) * h;
        if (RHS) r += p.rV1[c];
        dv[0] = r;
    }
    if (ok[1]) {  // V2 (I, J-1/2, K)
        const int m = c - sy;
        const T Pm = p.P[m];
        T r = mom2<T, G>(p.geo, p.d1, p.d2, p.d3, I, J, p.t22[m] - Pm, s22, p.t33[m] - Pm, s33,
                         p.t12[c - sy - sz], p.t12[c - 1 - sy - sz], p.t23[c - 1 - sy], p.t23[c - 1 - sy - sz]);
        if (RHS) r += p.rV2[c];
        dv[1] = r;
    }
    if (ok[2]) {  // V3 (I, J, K-1/2)
        const int m = c - sz;
        T r = mom3<T, G>(p.geo, p.d1, p.d2, p.d3, I, J, p.t33[m] - p.P[m], s33, p.t13[c - sy - sz], p.t13[c - 1 - sy - sz],
                         p.t23[c - 1 - sz], p.t23[c - 1 - sy - sz]);
        if (G == CART && GRAV) r -= p.g * (h * (p.rho[m] + p.rho[c]));
        if (RHS) r += p.rV3[c];
        dv[2] = r;
    }
}

// max |dV + rV| of the correction problem over the velocity nodes of block (bx, by, bz) into
// *red (inner stopping test); 32 x 8 threads, the body of k_velocity_norm and of its batched
// launch over many grids
template <typename T, int G>
__device__ __forceinline__ void velocity_norm_body(const KP<T>& p, int bx, int by, int bz, unsigned long long* red) {
    const int I = bx * blockDim.x + threadIdx.x + 1, J = by * blockDim.y + threadIdx.y + 1, K = bz + 1;
    const Dims& d = p.d;
    unsigned long long m = 0ULL;  // ordered bits of the running max (NaN propagates)
    if (I <= d.n1 - 1 && J <= d.n2 - 1 && K <= d.n3 - 1) {
        T dv[3];
        bool ok[3];
        momentum<T, G, false, true>(p, I, J, K, dv, ok);
        for (int f = 0; f < 3; ++f)
            if (ok[f]) m = umax64(m, ord_bits((double)dv[f]));
    }
    // block reduction over the 2D block
    for (int o = 16; o > 0; o >>= 1) m = umax64(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ unsigned long long sm[32];
    const int t = threadIdx.x + blockDim.x * threadIdx.y;
    const int lane = t & 31, w = t >> 5, nw = (blockDim.x * blockDim.y) >> 5;
    if (lane == 0) sm[w] = m;
    __syncthreads();
    if (w == 0) {
        m = lane < nw ? sm[lane] : 0ULL;
        for (int o = 16; o > 0; o >>= 1) m = umax64(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) atomicMax(red, m);
    }
}

template <typename T, int G>
__global__ void __launch_bounds__(256) k_velocity_norm(KP<T> p) {
    velocity_norm_body<T, G>(p, blockIdx.x, blockIdx.y, blockIdx.z, p.red);
}

// ---------------------------------------------------------------------------
// Boundary conditions.  A BC set is a list of stages run in order; the ops of
// one stage act on different fields across the faces normal to one axis, so
// they are independent.  Each op writes both faces of its field:
//   NEG     A[b] = -A[in]          COPY  A[b] = A[in]          ZERO  A[b] = 0
//   LIN     A[b] = (x_cd - c1)*c0  LIN2M A[b] = 2*(x_cd - c1)*c0 - A[in]
//   STRESS  normal-velocity ghost that makes the boundary cell divergence-free
//           (not in the reference)
// x_cd is the cell-centre coordinate of the node along axis cd.  In the
// homogeneous form (correction problem) constants vanish: LIN -> 0,
// LIN2M -> -A[in].
// BC_STRESS_SRC: BC_STRESS in a stage that also copies the two tangential fields
// into their ghost layer; it reads those fields at the copies' source cells
// instead of at the ghosts the copies are writing (the same values)
enum BcKind { BC_NEG = 0, BC_COPY = 1, BC_ZERO = 2, BC_LIN = 3, BC_LIN2M = 4, BC_STRESS = 5, BC_STRESS_SRC = 6 };
struct BcOp { int field; int kind; int cd; double c0, c1; int side; };  // side: -1 both faces, 0 low, 1 high
struct BcStage { int dim; int nops; BcOp op[3]; };
// The program as launched: stage D acts on axis D and has one op for every field f and side, op[D][f][side]; a
// stress op, BC_STRESS_SRC, is on the normal field (bc_closed checks it).  A launch runs the stages
// first .. last - 1, of which one at most has a stress op, or else it is a single stage.  Then the value of a
// ghost follows from entries that the launch does not write: undo the stages from the last to the
// first, each of which replaces a boundary index by an inner one.
struct BcFaceOp { int kind, cd; double c0, c1; };
struct BcProg { BcFaceOp op[3][3][2]; };

// V[f] at offset o, as a select between the three pointers
template <typename T>
__device__ __forceinline__ T vload(const KP<T>& p, int f, int o) { return (f == 0 ? p.V1 : (f == 1 ? p.V2 : p.V3))[o]; }
template <typename T>
__device__ __forceinline__ T* vfield(const KP<T>& p, int f) { return f == 0 ? p.V1 : (f == 1 ? p.V2 : p.V3); }

// one op with its coordinate factor looked up: applied to the inner value
template <typename T>
struct BcAct { int kind; T x, c0; };
template <typename T>
__device__ __forceinline__ BcAct<T> bc_act(const KP<T>& p, const BcFaceOp& op, int homog, int idx) {
    BcAct<T> a;
    a.kind = op.kind; a.x = T(0); a.c0 = T(0);
    if (op.kind == BC_LIN || op.kind == BC_LIN2M) {
        if (homog) {
            a.kind = op.kind == BC_LIN ? BC_ZERO : BC_NEG;
        } else {
            const T* xc = op.cd == 0 ? p.geo.x1c : (op.cd == 1 ? p.geo.x2c : p.geo.x3c);
            a.x = xc[idx] - T(op.c1);
            a.c0 = T(op.c0);
        }
    }
    return a;
}
template <typename T>
__device__ __forceinline__ T bc_apply(const BcAct<T>& a, T in) {
    switch (a.kind) {
        case BC_NEG: return -in;
        case BC_ZERO: return T(0);
        case BC_LIN: return a.x * a.c0;
        case BC_LIN2M: return T(2) * a.x * a.c0 - in;
        default: return in;
    }
}

__device__ __forceinline__ int bc_n(const Dims& d, int D) { return D == 0 ? d.n1 : (D == 1 ? d.n2 : d.n3); }

// undo the stages first .. S - 1 at index x of field f: x becomes the index of the value they start from, act[s]
// what stage s does to it.  Returns the stage whose stress op the entry is (x as that stage sees it), or -1.
template <typename T, int S>
__device__ __forceinline__ int bc_resolve(const KP<T>& p, const BcProg& q, int homog, int first, int f, int (&x)[3], BcAct<T> (&act)[S]) {
    int stop = -1;
#pragma unroll
    for (int D = S - 1; D >= 0; --D) {
        act[D].kind = BC_COPY;
        const int last = bc_n(p.d, D) - 1 + (f == D);
        const int side = x[D] == 0 ? 0 : (x[D] == last ? 1 : -1);
        if (stop >= 0 || side < 0 || D < first) continue;
        const BcFaceOp& op = q.op[D][f][side];
        if (op.kind == BC_STRESS_SRC) { stop = D; continue; }
        act[D] = bc_act(p, op, homog, op.cd == 0 ? x[0] : (op.cd == 1 ? x[1] : x[2]));
        x[D] = side == 0 ? 1 : last - 1;
    }
    return stop;
}

// the divergence-free ghost of stage D at index x, from values after the stages first .. D - 1 (none with a stress op)
template <typename T, int G, int D>
__device__ __forceinline__ T bc_stress(const KP<T>& p, const BcProg& q, int homog, int first, const int (&x)[3]) {
    const Dims& d = p.d;
    const int n = bc_n(d, D), side = x[D] == 0 ? 0 : 1;
    const int cell = side == 0 ? 0 : n - 1, src = side == 0 ? 1 : n - 2, in = side == 0 ? 1 : n - 1;
    constexpr int A = D == 0 ? 1 : 0, B = D == 2 ? 1 : 2;  // tangential axes
    // inside normal face, low and high faces along A and B: all five resolved, then loaded together
    const CellMetric<T> c = cell_metric<T, G>(p, D == 0 ? cell : x[0], D == 1 ? cell : x[1]);
    T v[5];
    BcAct<T> act[5][D + 1];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
        const int f = m == 0 ? D : (m <= 2 ? A : B);
        int y[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) y[a] = a == D ? (m == 0 ? in : src) : x[a] + ((m == 2 && a == A) || (m == 4 && a == B) ? 1 : 0);
        bc_resolve<T, D + 1>(p, q, homog, first, f, y, act[m]);  // (stage D leaves it: y[D] is inside)
        v[m] = vload(p, f, y[0] + d.sy * y[1] + d.sz * y[2]);
    }
#pragma unroll
    for (int m = 0; m < 5; ++m)
#pragma unroll
        for (int s = 0; s < D; ++s) v[m] = bc_apply(act[m][s], v[m]);
    if (D == 0) return div_ghost<T, G, 0>(c, p.d1, side, v[0], v[0], v[1], v[2], v[3], v[4]);
    if (D == 1) return div_ghost<T, G, 1>(c, p.d1, side, v[1], v[2], v[0], v[0], v[3], v[4]);
    return div_ghost<T, G, 2>(c, p.d1, side, v[1], v[2], v[3], v[4], v[0], v[0]);
}

// face point (u, v) of stage D: both faces of every field, loads first.  Other stages of the launch do not touch
// what it reads: (u, v) is inside along the other two axes, or the launch is this stage alone
template <typename T, int G, int D>
__device__ __forceinline__ void bc_face(const KP<T>& p, const BcProg& q, int homog, int u, int v) {
    const Dims& d = p.d;
    const int x0 = D == 0 ? 0 : u, x1 = D == 1 ? 0 : (D == 0 ? u : v), x2 = D == 2 ? 0 : v;
    const int base = x0 + d.sy * x1 + d.sz * x2, step = D == 0 ? 1 : (D == 1 ? d.sy : d.sz);
    const int nu = D == 0 ? d.n2 : d.n1, nv = D == 2 ? d.n2 : d.n3, du = D == 0 ? 1 : 0, dv = D == 2 ? 1 : 2, n = bc_n(d, D);
    T val[3][2];
    BcAct<T> act[3][2];
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        const int last = n - 1 + (f == D);
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const BcFaceOp& op = q.op[D][f][side];
            act[f][side].kind = -1;
            if (u >= nu + (f == du) || v >= nv + (f == dv) || op.kind == BC_STRESS_SRC) continue;
            val[f][side] = vload(p, f, base + (side == 0 ? 1 : last - 1) * step);
            act[f][side] = bc_act(p, op, homog, op.cd == D ? (side == 0 ? 0 : last) : (op.cd == 0 ? x0 : (op.cd == 1 ? x1 : x2)));
        }
    }
#pragma unroll
    for (int f = 0; f < 3; ++f)
#pragma unroll
        for (int side = 0; side < 2; ++side)
            if (act[f][side].kind >= 0) vfield(p, f)[base + (side == 0 ? 0 : n - 1 + (f == D)) * step] = bc_apply(act[f][side], val[f][side]);
    if (u >= nu || v >= nv) return;
    for (int side = 0; side < 2; ++side) {
        if (q.op[D][D][side].kind != BC_STRESS_SRC) continue;
        const int cell = side == 0 ? 0 : n - 1, ci = base + (side == 0 ? 1 : n - 1) * step, ct = base + (side == 0 ? 1 : n - 2) * step;
        const CellMetric<T> m = cell_metric<T, G>(p, D == 0 ? cell : x0, D == 1 ? cell : x1);
        T g;
        if (D == 0)
            g = div_ghost<T, G, 0>(m, p.d1, side, p.V1[ci], p.V1[ci], p.V2[ct], p.V2[ct + d.sy], p.V3[ct], p.V3[ct + d.sz]);
        else if (D == 1)
            g = div_ghost<T, G, 1>(m, p.d1, side, p.V1[ct], p.V1[ct + 1], p.V2[ci], p.V2[ci], p.V3[ct], p.V3[ct + d.sz]);
        else
            g = div_ghost<T, G, 2>(m, p.d1, side, p.V1[ct], p.V1[ct + 1], p.V2[ct], p.V2[ct + d.sy], p.V3[ci], p.V3[ci]);
        vfield(p, D)[base + (side == 0 ? 0 : n) * step] = g;
    }
}

constexpr int BC_SM_PLANES = 4;  // planes of ηSM per thread

// Stages first .. last - 1 in one launch.  A single stage: blocks of face points.  Otherwise blocks z < last - first
// take the points of their stage's faces that are inside along the other axes, and the blocks of the last
// z everything near an edge of the box: a warp per 32 points of a line (field, direction of the line, places of the
// other two indices) or per field's corners, each ghost undone to entries that the launch does not write.
// Ghosts of a later stage are left to it.
// (One stress op at most: its inputs then resolve to values that need no other stress ghost.)
// Blocks past those, where a launch has them: ηSM of the next iteration (its η is final, and no boundary value enters).
// Bound by latency, of the launch and of loads and stores in a row.  us per iteration with a launch for each
// stage and each op's load behind the store before, and so: FP64 70 x 5 x 5 27.4 and 19.4,
// FP32 95 x 79 x 67 42.1 and 33.9, FP64 63^3 126 and 117.5.
template <typename T, int G>
__global__ void __launch_bounds__(128) k_bc(const __grid_constant__ KP<T> p, const __grid_constant__ BcProg q, int homog, int first, int last, int early) {
    pdl_wait();
    if (early) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    const Dims& d = p.d;
    const int z = first + blockIdx.z;
    const bool single = last - first == 1;
    const int nz = single ? 1 : last - first + 1;
    if (blockIdx.z >= nz) {
        const int nt = 32 * blockDim.y, cols = (d.n1 * d.n2 + nt - 1) / nt;
        const int lin = ((blockIdx.z - nz) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        const int col = lin % cols * nt + threadIdx.y * 32 + threadIdx.x, k0 = lin / cols * BC_SM_PLANES;
        const int i = col % d.n1, j = col / d.n1;
#pragma unroll
        for (int k = 0; k < BC_SM_PLANES; ++k) maxloc_body(p, (int)(G == CART), i, j, k0 + k);
        return;
    }
    if (z < last) {
        const int u = blockIdx.x * 32 + threadIdx.x, v = blockIdx.y * blockDim.y + threadIdx.y;
        if (!single && (u < 1 || v < 1 || u > bc_n(d, z == 0 ? 1 : 0) - 2 || v > bc_n(d, z == 2 ? 1 : 2) - 2)) return;
        if (z == 0) bc_face<T, G, 0>(p, q, homog, u, v);
        else if (z == 1) bc_face<T, G, 1>(p, q, homog, u, v);
        else bc_face<T, G, 2>(p, q, homog, u, v);
        return;
    }
    const int w0 = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.y + threadIdx.y, nw = gridDim.x * gridDim.y * blockDim.y;
    const int per = (max(d.n1, max(d.n2, d.n3)) + 29) / 32;  // warps of a line's n - 2 inner points
    for (int w = w0; w < 3 + 81 * per; w += nw) {
        int f = w, ax = 0, t = 0, b, c;
        if (w < 3) {  // corners
            if (threadIdx.x >= 27) continue;
            const int a = threadIdx.x % 3;
            b = threadIdx.x / 3 % 3;
            c = threadIdx.x / 9;
            if (a == 2 && f != 0) continue;
            t = a == 0 ? 0 : d.n1 - 2 + a;
        } else {
            const int line = (w - 3) / per;
            f = line / 27; ax = line / 9 % 3; b = line / 3 % 3; c = line % 3;
            t = 1 + ((w - 3) % per) * 32 + threadIdx.x;
            if (t > bc_n(d, ax) - 2) continue;
        }
        const int B = ax == 0 ? 1 : 0, C = ax == 2 ? 1 : 2;
        if ((b == 2 && f != B) || (c == 2 && f != C)) continue;
        const int xb = b == 0 ? 0 : bc_n(d, B) - 2 + b, xc = c == 0 ? 0 : bc_n(d, C) - 2 + c;
        int x[3] = {ax == 0 ? t : xb, ax == 1 ? t : (ax == 0 ? xb : xc), ax == 2 ? t : xc};
        bool ghost = false, later = false;
#pragma unroll
        for (int D = 0; D < 3; ++D) {
            const bool g = x[D] == 0 || x[D] == bc_n(d, D) - 1 + (f == D);
            if (D >= last) later = later || g;
            else if (D >= first) ghost = ghost || g;
        }
        if (!ghost || later) continue;
        const int at = x[0] + d.sy * x[1] + d.sz * x[2];
        BcAct<T> act[3];
        const int stop = bc_resolve<T, 3>(p, q, homog, first, f, x, act);
        T v;
        if (stop < 0) v = vload(p, f, x[0] + d.sy * x[1] + d.sz * x[2]);
        else if (stop == 0) v = bc_stress<T, G, 0>(p, q, homog, first, x);
        else if (stop == 1) v = bc_stress<T, G, 1>(p, q, homog, first, x);
        else v = bc_stress<T, G, 2>(p, q, homog, first, x);
#pragma unroll
        for (int s = 0; s < 3; ++s) v = bc_apply(act[s], v);
        vfield(p, f)[at] = v;
    }
}

// ---------------------------------------------------------------------------
// P_out = P except on the boundary cells of the normal-stress BC, where
// P_out = τ_nn - σ_bc from the given stresses (residual evaluation)
template <typename T>
__global__ void k_traction_pressure(KP<T> p, T* __restrict__ Pout) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
    const Dims& d = p.d;
    if (i >= d.n1 || j >= d.n2 || k >= d.n3) return;
    const int c = i + d.sy * j + d.sz * k;
    T P = p.P[c];
    if (p.traction) traction_pressure(j, k, d.n2, d.n3, p.t22[c], p.t33[c], p.sig2, p.sig3, P);
    if (p.fs && i == d.n1 - 1) P = fs_pressure(p.t11[c], p.top_load ? p.top_load[c] : T(0), p.fs_kappa, p.V1[c], p.V1[c + 1]);
    Pout[c] = P;
}

// ---------------------------------------------------------------------------
// reductions: max|a| (or max|a-b|) over n entries into red[slot], as the ordered
// bits of ord_bits (a NaN entry makes the result NaN, as Julia's maximum(abs.(.)))
// block-wide max of ordered bits, one atomicMax per block
__device__ __forceinline__ void block_max_to(unsigned long long v, unsigned long long* slot) {
    for (int o = 16; o > 0; o >>= 1) v = umax64(v, __shfl_xor_sync(0xffffffffu, v, o));
    __shared__ unsigned long long sm[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sm[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < (int)(blockDim.x >> 5) ? sm[lane] : 0ULL;
        for (int o = 16; o > 0; o >>= 1) v = umax64(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) atomicMax(slot, v);
    }
}

// The maxima of up to 8 fields in one launch, field blockIdx.y: max|a| into red[slot], and max|a - b| into
// red[slot_d] where there is a b; slot_d = kLeast: the least positive a, as the greatest of its inverted bits.  A launch per maximum and per snapshot copy cost a check as much as several iterations
// of a small grid: 200 FP64 iterations at 70 x 5 x 5 with a check every 10 took 4.24 ms with them, 3.42 with this
// and k_copy3; the FP64 residual of a 47 x 31 x 39 grid 73 and 37 us.
template <typename T>
struct MaxItem { const T *a, *b; int slot, slot_d; };
template <typename T>
struct MaxList { MaxItem<T> f[8]; };
constexpr int kLeast = -1;
template <typename T>
__global__ void __launch_bounds__(256) k_maxabs(const __grid_constant__ MaxList<T> list, long long n, unsigned long long* red) {
    pdl_enter_small();
    const MaxItem<T>& f = list.f[blockIdx.y];
    const T *a = f.a, *b = f.b;
    unsigned long long m = 0ULL, e = 0ULL;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const T x = a[q];
        if (f.slot_d == kLeast) {
            const long long v = __double_as_longlong((double)x);
            m = umax64(m, v > 0 ? ~(unsigned long long)v : 0ULL);
            continue;
        }
        m = umax64(m, ord_bits((double)x));
        if (b) e = umax64(e, ord_bits((double)x - (double)b[q]));
    }
    block_max_to(m, red + f.slot);
    if (!b) return;
    __syncthreads();  // (the scratch of the first reduction)
    block_max_to(e, red + f.slot_d);
}

// dst[f] = src[f], f = blockIdx.y
template <typename T>
__global__ void __launch_bounds__(256) k_copy3(T* d0, T* d1, T* d2, const T* s0, const T* s1, const T* s2, long long n) {
    pdl_enter_small();
    T* d = blockIdx.y == 0 ? d0 : (blockIdx.y == 1 ? d1 : d2);
    const T* s = blockIdx.y == 0 ? s0 : (blockIdx.y == 1 ? s1 : s2);
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) d[q] = s[q];
}

// ---------------------------------------------------------------------------
// elementwise helpers over the whole box
template <typename TD, typename TS>
__global__ void k_convert(TD* __restrict__ dst, const TS* __restrict__ src, long long n) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) dst[q] = (TD)src[q];
}
// dst += (double)src
template <typename TS>
__global__ void k_add_widen(double* __restrict__ dst, const TS* __restrict__ src, long long n) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) dst[q] += (double)src[q];
}

// A field in the reference layout (dense e0 x e1 x e2 doubles, x1 fastest) <-> its
// entries in the padded box (strides 1, sy, sz).  Launch: grid (ceil(e0/blockDim.x),
// e1, e2); one entry per thread, consecutive threads on consecutive x1 entries on
// both sides.  The host copies whole dense fields in one transfer and these kernels
// do the re-pitching on the device.
template <typename T>
__device__ __forceinline__ T from_double(double v) { return (T)v; }
template <>
__device__ __forceinline__ uint8_t from_double<uint8_t>(double v) { return v != 0.0 ? 1 : 0; }

template <typename T>
__global__ void k_unpack(T* __restrict__ box, const double* __restrict__ dense, int e0, int e1, int sy, int sz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= e0) return;
    const int j = blockIdx.y, k = blockIdx.z;
    box[i + (long long)sy * j + (long long)sz * k] = from_double<T>(dense[i + (long long)e0 * (j + (long long)e1 * k)]);
}
template <typename T>
__global__ void k_pack(double* __restrict__ dense, const T* __restrict__ box, int e0, int e1, int sy, int sz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= e0) return;
    const int j = blockIdx.y, k = blockIdx.z;
    dense[i + (long long)e0 * (j + (long long)e1 * k)] = (double)box[i + (long long)sy * j + (long long)sz * k];
}

}  // namespace sph
