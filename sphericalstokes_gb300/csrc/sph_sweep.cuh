// Fused FP32 PT sweep: compute_P! and compute_V! of one PT iteration in one
// launch (SphericalStokes_diapir.jl:209-241, :287-329), fed by TMA, two
// x1-adjacent points per thread in paired FP32 arithmetic.
//
// A block owns a 32 x 14 column of cells in (x1, x2) and marches along x3 over a
// chunk of planes.  Per plane K: stage 1 updates P, τ11..τ33 (cells) and τ12,
// τ13, τ23 (edges) on the tile plus a one-point halo on the low x1 / x2 sides,
// stores the owned points and leaves σ, the edge stresses and DT_R / 2 in shared
// memory; after a block barrier the velocities of plane K follow from the
// stresses of planes K-1 and K.  Every state field is read once and written once
// per sweep (old and new state are different buffers).
//
// MODE 1: correction problem of the mixed-precision solve (right-hand sides rP,
// rV; η and ηSM frozen; homogeneous boundary data).  MODE 0: reference iteration
// (ρg body force).
//
// Bound: HBM (104 B per cell and sweep).  What the layout is for:
// * Issue slots.  A thread owns a pair of points, so arithmetic is FFMA2 / FADD2 /
//   FMUL2, shared-memory and global accesses are 8 bytes wide, and the per-plane
//   bookkeeping is shared by two cells.  A difference a - b is one FFMA2 with the
//   constant -1 (a paired add cannot negate an operand).  Of η and ηSM, what plane K+1
//   contributes to the stencils of plane K is what it needs of itself at the next step:
//   the pair's values and their sums over two cells (6 pairs) are carried in registers, with
//   the stresses of plane K that the velocities of plane K+1 want, and each plane of η and
//   ηSM is read from shared memory once; the velocities of a plane are read at both steps.
// * Copies in flight.  Stage 1 of plane K reads the input slots of planes K and K+1, so that
//   three slots (12.5 KB each) keep one to two planes in flight, with the old state and the
//   right-hand sides in two (22 KB each); the warp that computes the halo points has no velocities to
//   update and issues them (7 four-dimensional boxes per plane: fields of a slab are equally spaced).
// * 14 rows, because 7 warps of owned points and one of halo points (31 pairs) make four
//   warps per scheduler at two blocks per SM, which leaves 128 registers to each thread:
//   16 rows need a ninth warp, five warps on some schedulers, 96 registers and spills.
// * Uniform paths.  Faces, masks and ghosts are bits set once per pair; a warp whose points
//   are all inside takes the path without masks (a vote at the start of the block), ghosts on
//   x1 travel with the pair's own store, and the divergence-free x2 ghosts and the loaded x2
//   faces are paired arithmetic: no plane diverges except the first and last of the grid and
//   the rows on an x1 face with such a ghost.
// Measured on a GB300, us per sweep with its boundary velocities (before: one cell per
// thread, 32 x 8 tiles, 30 warps per SM, x2 / x3 ghosts by two to four BC launches):
// 255^3 304 (375; 5.7 TB/s of the algorithmic bytes, 0.85 of the copy rate),
// 511 x 255 x 255 with a free surface 607 (732), 131 x 117 x 101 44.1 (65.0),
// 63^3 11.8 (19.1), 47 x 31 x 39 Cartesian 6.2 (14.5).  At 255^3 316 warp instructions
// per 32 cells (608).  The same copies and stores without the arithmetic take 285 us
// (the tiles' halos and 10 + 10 streams cost 10 % of the copy rate): memory bound there.  The
// smallest grids are one wave of blocks: the latency of a few planes and the launch.
//
// Thread roles (8 warps): warp w < 7, lane l: row b = 2w + l/16 + 1, points
// a = 2(l%16) + 1, +2, i.e. cells (x0 + 2(l%16) + {0,1}, y0 + b - 1), and the
// velocity nodes of the same indices.  Warp 7: lanes 0..15 the halo row b = 0,
// lanes 16..30 the halo column a = 0 of the rows b = l - 16 (pairs (-1, 0), of which
// the first point is discarded).  Point (a, b) is the cell (x0 - 1 + a, y0 - 1 + b).
//
// Boundary velocities of the correction problem (SweepOut::gmask, smask): the
// thread that computes a node next to a face also stores the face's ghosts, and
// the divergence-free normal ghosts are evaluated by the one stencil that reads
// them (the strain rates of the boundary cell; the edge stencils read interior
// normal velocities only) from the cell's other face velocities.  On edges and
// corners such a ghost is the copy of the one at the nearest interior cell along
// the later axes, evaluated from global memory.  No BC launch follows a sweep.
#pragma once
#include <cuda.h>

#include <type_traits>

#include "sph_core.cuh"

namespace sph {

template <typename T>
struct SweepOut {
    T *P, *V1, *V2, *V3, *t11, *t22, *t33, *t12, *t13, *t23;
    // The homogeneous BC program in closed form (build_ghosts).  Bit 6 dim + 2 field + side of
    // gmask: the ghost of `field` on that face of axis `dim` is gf[3 dim + field] x its interior
    // neighbour, written with the new values (products on edges and corners, as the stages leave
    // them).  Bit 2 dim + side of smask: the normal ghost of that face makes the boundary cell
    // divergence-free; it is not stored but evaluated where the next sweep reads it.
    int gmask, smask;
    float gf[9];
    float small;  // 2^-126 / min(1, GSDT/ηSM, KBDT/ηSM)
    // scalars of the sweep as pairs (operands of the paired instructions straight from constant memory)
    float2 d1, d1q, d2, gsc, kbc, nkbc, vp, third, half;  // d1, d1 / 4, d2, GSDT/ηSM, ±KBDT/ηSM, vpdt² / 2, -1/3, -1/2
};

// ---------------------------------------------------------------------------
// TMA and mbarrier helpers
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// bounded wait on the phase with the given parity; false if the bound ran out.
// Each try_wait suspends the thread until the phase completes or the suspend hint
// (kMbarSuspendNs) passes, so a waiting warp does not re-issue polls; kMbarMaxPolls
// of them bound the wait to about 2 s.  The bound is a count of polls, so the wait
// ends whatever the hint does.
constexpr unsigned kMbarSuspendNs = 200000;
constexpr int kMbarMaxPolls = 10000;
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int max_polls = kMbarMaxPolls,
                                          unsigned suspend_ns = kMbarSuspendNs) {
    const unsigned a = smem_u32(bar);
    for (int it = 0; it < max_polls; ++it) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(a), "r"(parity), "r"(suspend_ns) : "memory");
        if (done) return true;
    }
    return false;
}

// Self-test of the bounded-wait error path of the TMA sweeps: one block waits on an
// mbarrier that nothing completes (initialised for one arrival, never arrived at, no
// copy issued), with the sweeps' wait at max_polls polls of suspend_ns; when the
// bound runs out it records 1 in *err as the sweep kernels do, and returns.
__global__ void k_wait_selftest(int* err, int max_polls, unsigned suspend_ns) {
    __shared__ unsigned long long bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && !mbar_wait(&bar, 0u, max_polls, suspend_ns)) atomicExch(err, 1);
}
// box of a map over (x1, x2, x3, field) starting at (x, y, z, 0)
__device__ __forceinline__ void tma_load4d(float* dst, const CUtensorMap* map, int x, int y, int z, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(0), "r"(smem_u32(bar))
        : "memory");
}

// ---------------------------------------------------------------------------
// paired FP32 arithmetic
__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return reinterpret_cast<float2&>(r);
}
// fast quotient per lane: the approximate reciprocal (1 ulp; subnormal inputs and results are zero)
// times a.  __fdividef costs several instructions more per lane, for subnormal operands.
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 div2(float2 a, float2 b) { return __fmul2_rn(a, make_float2(rcp_approx(b.x), rcp_approx(b.y))); }
// The divisors of the sweep are GSDT, KBDT or more: subnormal only where ηSM is below `small` (SweepOut).  LIFT: there both
// operands are multiplied by 2^24 first, which changes no other bit of a quotient.
template <bool LIFT>
__device__ __forceinline__ float2 div2(float2 a, float2 b, float2 etaSM, float small) {
    if (!LIFT) return div2(a, b);
    const float2 c = make_float2(etaSM.x < small ? 16777216.f : 1.f, etaSM.y < small ? 16777216.f : 1.f);
    return div2(mul2(a, c), mul2(b, c));
}
__device__ __forceinline__ float2 keep2(float2 x, bool m0, bool m1) { return make_float2(m0 ? x.x : 0.f, m1 ? x.y : 0.f); }

// stores at a 32-bit unsigned byte offset from a field's base: the address is the
// base plus a zero-extended register, with no 64-bit index arithmetic per store
__device__ __forceinline__ void st_at(float* base, unsigned byte_off, float v) {
    *reinterpret_cast<float*>(reinterpret_cast<char*>(base) + byte_off) = v;
}
__device__ __forceinline__ void st_pair(float* base, unsigned byte_off, float2 v) {
    *reinterpret_cast<float2*>(reinterpret_cast<char*>(base) + byte_off) = v;
}
__device__ __forceinline__ void st_pair(float* base, unsigned byte_off, float2 v, bool m0, bool m1) {
    if (m0 && m1) {
        st_pair(base, byte_off, v);
    } else {
        if (m0) st_at(base, byte_off, v.x);
        if (m1) st_at(base, byte_off + 4u, v.y);
    }
}

// ---------------------------------------------------------------------------
constexpr int SWX = 32, SWY = 14;          // owned tile (cells) per block
constexpr int SW_NT = 256;                 // threads per block
constexpr int SI_X = 40, SI_Y = SWY + 2;   // input boxes (V, η, ηSM), origin (x0 - 4, y0 - 1)
constexpr int SO_X = 36, SO_Y = SWY + 1;   // old-state boxes (P, τ, rP | ρ), same origin
constexpr int SR_X = 34;                   // row of the shared stresses: a = -1 .. 32 at a + 1
constexpr int SI_N = SI_X * SI_Y, SO_N = SO_X * SO_Y, SR_N = SR_X * SO_Y, SV_N = SWX * SWY;

// tensor maps of one arrangement of the buffers
enum SweepMap { SM_V = 0, SM_ETA, SM_ETASM, SM_P, SM_TAU, SM_RP, SM_RHO, SM_RV, SM_COUNT };
struct SweepMaps { alignas(128) CUtensorMap m[SM_COUNT]; };

constexpr int pad128(int floats) { return (floats + 31) / 32 * 32; }
struct SweepSmem {
    alignas(128) float in[3][5 * SI_N];       // V1, V2, V3, η, ηSM
    alignas(128) float P[2][pad128(SO_N)];
    alignas(128) float tau[2][pad128(6 * SO_N)];
    alignas(128) float rp[2][pad128(SO_N)];   // rP | ρ
    alignas(128) float rv[2][pad128(3 * SV_N)];
    alignas(16) float q[4][SR_N];             // σ11, σ22, σ33, DT_R / 2 of plane K
    alignas(16) float e[2][3][SR_N];          // τ12, τ13, τ23 of planes K-1, K
    float2 mom[4][SW_NT - 32];                // spherical: m1_d3, m1_t, m2_d3, m2_n of each thread
    unsigned long long bar_s[2], bar_v[2], bar_0;
};
inline size_t sweep_smem_bytes() { return sizeof(SweepSmem); }

// Coefficients of a pair of points: the metric factors of sph_core.cuh multiplied out with the
// spacings once per thread, so that each update is a short chain of FMAs (2 (x h) = x,
// 3 (x h) = 1.5 x: the same values up to FP32 rounding).
struct SweepCoef {
    // cell, with Σ the sums of the two face velocities: div = d1 Δ1 + a2 Δ2 + a3 Δ3 + 2 e1 Σ1
    // (cylindrical: e1 Σ1) + e2 Σ2, D22 = a2 Δ2 + e1 Σ1 - div/3, D33 = a3 Δ3 + e1 Σ1 (spherical) + e2 Σ2 - div/3
    float2 a2, a3, e1, e2;
    // quarters of the engineering shear rates (the edge update wants D / 4)
    float2 e12_d2, e12_h;          // τ12: iRh d2 / 4, -iRh / 8
    float2 e13_d3;                 // τ13: iRh iSc1 d3 / 4 (and -iRh / 8)
    float2 e23_d2, e23_d3, e23_h;  // τ23: iRc1 d2 / 4, iRc1 iSh d3 / 4, -iRc1 ctH / 8
    float2 m1_i, m1_d3, m1_t;      // V1: iR1 (Cartesian: 1), iR1 iS1 d3, iR1 ct1 / 2
    float2 m2_d3, m2_s, m2_n;      // V2 (and a2): iR2 iS2 d3, shear and normal-stress metric terms; V3: a2, a3, m2_s or e1, e2
};
template <int G>
__device__ __forceinline__ SweepCoef sweep_coef(const Geo<float>& geo, float d2, float d3, int xa, int y, int n1, int n2) {
    SweepCoef c;
    float* out = reinterpret_cast<float*>(&c);
    for (int l = 0; l < 2; ++l) {
        const int x = xa + l;
        const CellMetric<float> cm = cell_metric_t<float, G>(geo, d2, d3, clampi(x, 0, n1 - 1), clampi(y, 0, n2 - 1));
        const EdgeMetric<float> e = edge_metric<float, G>(geo, x, y, n1, n2);
        const MomMetric<float> m = mom_metric<float, G>(geo, x, y, n1, n2);
        const float v[16] = {cm.a2, cm.a3, 0.5f * cm.e1, 0.5f * cm.e2,
                             0.25f * e.iRh * d2, -0.125f * e.iRh,
                             0.25f * (G == SPH ? e.iRh * e.iSc1 * d3 : d3),
                             0.25f * e.iRc1 * d2, 0.25f * (G == SPH ? e.iRc1 * e.iSh * d3 : d3), -0.125f * e.iRc1 * e.ctH,
                             m.iR1, G == SPH ? m.iR1 * m.iS1 * d3 : d3, 0.5f * m.iR1 * m.ct1,
                             G == SPH ? m.iR2 * m.iS2 * d3 : d3, G == SPH ? 1.5f * m.iR2 : m.iR2, 0.5f * m.iR2 * m.ct2};
        for (int i = 0; i < 16; ++i) out[2 * i + l] = v[i];
    }
    return c;
}

// Boundary work of the sweep, which few points run:
// the divergence-free ghosts (smask) of cell (x, y, k) among its six face velocities v; the cell's
// metric from its sweep coefficients (exact: they are powers of two times the metric factors)
template <int G>
__device__ __forceinline__ void sweep_fill_ghosts(const KP<float>* pp, int smask, int x, int y, int k, float a2, float a3, float e1, float e2,
                                               float* v) {
    const KP<float>& p = *pp;
    const Dims& d = p.d;
    const int n1 = d.n1, n2 = d.n2, n3 = d.n3;
    const int s = smask & ((x == 0 ? 1 : 0) | (x == n1 - 1 ? 2 : 0) | (y == 0 ? 4 : 0) | (y == n2 - 1 ? 8 : 0) | (k == 0 ? 16 : 0) |
                           (k == n3 - 1 ? 32 : 0));
    CellMetric<float> m;
    m.a2 = a2; m.a3 = a3; m.c1 = (G == SPH ? 4.f : 2.f) * e1; m.c2 = 2.f * e2; m.e1 = m.e1b = m.e2 = 0.f;
    // ghost of axis D at cell (x, j, kk) from global memory (edges and corners)
    auto at = [&](auto axis, int side, int j, int kk) {
        constexpr int D = decltype(axis)::value;
        const int c = x + d.sy * j + d.sz * kk;
        return div_ghost<float, G, D>(cell_metric_t<float, G>(p.geo, p.d2, p.d3, x, j), p.d1, side, p.V1[c], p.V1[c + 1], p.V2[c],
                                      p.V2[c + d.sy], p.V3[c], p.V3[c + d.sz]);
    };
    const int kc = clampi(k, 1, n3 - 2), jc = clampi(y, 1, n2 - 2);
    if (s & 3) {
        const int side = s & 1 ? 0 : 1;
        const float g = (jc != y || kc != k) ? at(std::integral_constant<int, 0>{}, side, jc, kc)
                                             : div_ghost<float, G, 0>(m, p.d1, side, v[0], v[1], v[2], v[3], v[4], v[5]);
        if (side) v[1] = g;
        else v[0] = g;
    }
    if (s & 12) {
        const int side = s & 4 ? 0 : 1;
        const float g = kc != k ? at(std::integral_constant<int, 1>{}, side, y, kc)
                                : div_ghost<float, G, 1>(m, p.d1, side, v[0], v[1], v[2], v[3], v[4], v[5]);
        if (side) v[3] = g;
        else v[2] = g;
    }
    if (s & 48) {
        const int side = s & 16 ? 0 : 1;
        const float g = div_ghost<float, G, 2>(m, p.d1, side, v[0], v[1], v[2], v[3], v[4], v[5]);
        if (side) v[5] = g;
        else v[4] = g;
    }
}
// maps: tensor maps among the launch's parameters, or in global memory after a tensor-map fence
// LIFT: divisors may be subnormal (div2).  MODE 1 has fixed η and its least one is known to the host (Ctx::small32); the η of
// MODE 0 changes, and it always lifts.  us per sweep without and with: 63^3 11.80 and 12.07, 255^3 304.4 and 309.0 (by a branch to __fdividef 12.20
// and 317.1; both marches in one kernel, chosen by a word in memory, 12.19 and 307.7).
template <int G, int MODE, bool LIFT>
__device__ __forceinline__ void sweep_body(const KP<float>& p, const SweepOut<float>& o, int kchunk, const CUtensorMap* __restrict__ maps,
                                           int* __restrict__ err, int bx, int by, int bz) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    SweepSmem& S = *reinterpret_cast<SweepSmem*>(smem_raw);

    const Dims d = p.d;
    const int tid = threadIdx.x;
    const int x0 = bx * SWX, y0 = by * SWY;
    const int kA = bz * kchunk;
    const int kB = min(kA + kchunk, d.n3);
    const int n1 = d.n1, n2 = d.n2, n3 = d.n3;
    if (kA >= kB) return;
    const int k0 = kA > 0 ? kA - 1 : 0;  // first plane of stage 1

    const int warp = tid >> 5, lane = tid & 31;
    const bool halo = warp == SWY / 2;
    const bool issuer = tid == SW_NT - 32;
    if (issuer) {
        for (int i = 0; i < 2; ++i) { mbar_init(&S.bar_s[i], 1); mbar_init(&S.bar_v[i], 1); }
        mbar_init(&S.bar_0, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();

    // ---- copies (issuer only)
    auto issue_in = [&](int z, unsigned long long* bar) {
        float* t = S.in[(z - k0) % 3];
        tma_load4d(t, maps + SM_V, x0 - 4, y0 - 1, z, bar);
        tma_load4d(t + 3 * SI_N, maps + SM_ETA, x0 - 4, y0 - 1, z, bar);
        tma_load4d(t + 4 * SI_N, maps + SM_ETASM, x0 - 4, y0 - 1, z, bar);
    };
    // what stage 1 of plane k reads: inputs of plane k + 1, old state (and rP) of plane k
    auto issue_stage = [&](int k) {
        const int par = (k - k0) & 1;
        unsigned long long* bar = &S.bar_s[par];
        mbar_expect_tx(bar, 4 * (5 * SI_N + (MODE == 1 ? 8 : 7) * SO_N));
        issue_in(k + 1, bar);
        tma_load4d(S.P[par], maps + SM_P, x0 - 4, y0 - 1, k, bar);
        tma_load4d(S.tau[par], maps + SM_TAU, x0 - 4, y0 - 1, k, bar);
        if (MODE == 1) tma_load4d(S.rp[par], maps + SM_RP, x0 - 4, y0 - 1, k, bar);
    };
    // what the velocities of plane k read besides: rV (MODE 1) or ρ (MODE 0)
    auto issue_rhs = [&](int k) {
        const int par = (k - k0) & 1;
        unsigned long long* bar = &S.bar_v[par];
        mbar_expect_tx(bar, 4 * (MODE == 1 ? 3 * SV_N : SO_N));
        if (MODE == 1) tma_load4d(S.rv[par], maps + SM_RV, x0, y0, k, bar);
        else tma_load4d(S.rp[par], maps + SM_RHO, x0 - 4, y0 - 1, k, bar);
    };
    // false once a bounded wait ran out: from then on the waiting warp neither waits nor issues
    // copies, so the block finishes its march on whatever the tiles hold and exits
    bool ok = true;
    unsigned ph = 0;  // parity bits: bar_s 0, 1; bar_v 2, 3
    auto wait = [&](unsigned long long* bar, int bit) {
        if (!ok) return;
        ok = mbar_wait(bar, (ph >> bit) & 1u);
        ph ^= 1u << bit;
    };

    pdl_wait();  // (nothing before this reads what the preceding sweep writes)
    if (issuer) {
        mbar_expect_tx(&S.bar_0, 4 * 5 * SI_N);
        issue_in(k0, &S.bar_0);
        issue_stage(k0);
        if (k0 + 1 < kB) issue_stage(k0 + 1);
        issue_rhs(kA);
    }

    // ---- per-thread constants of the whole march (point l of the pair: l = 0, 1)
    const int lp = lane & 15;
    const bool col = halo && lane >= 16;  // halo column
    const int a = col ? -1 : 2 * lp + 1;
    const int b = halo ? (col && lane < 31 ? lane - 16 : 0) : 2 * warp + (lane >> 4) + 1;
    const int x = x0 - 1 + a, y = y0 - 1 + b;
    const bool yin = y >= 0 && y < n2 && !(halo && lane == 31);
    const bool in0 = yin && !col && x < n1, in1 = yin && x + 1 >= 0 && x + 1 < n1;  // (!col: x >= 0)
    const int iin = b * SI_X + a + 3, iold = b * SO_X + a + 3, ist = b * SR_X + a + 1;
    const SweepCoef C = sweep_coef<G>(p.geo, p.d2, p.d3, x, y, n1, n2);
    const int I = x, J = y;  // velocity nodes (I, J), (I + 1, J) of the owned points
    const int gxy = x + d.sy * y;
    // what holds for this pair's points whatever the plane, one bit each (point l: bit + l)
    enum { IN_ = 0, E12_ = 2, E13_ = 4, E23_ = 6,  // inside the grid: cells, edges
           M_ = 8,        // entries of V1 (+2: V2, +4: V3) this pair writes: nodes, and x1 ghosts within the pair
           X_ = 14,       // V1 (+1, +2): the high x1 ghost follows the pair's second point
           XLO = 17,      // the pair's first point is the low x1 ghost
           XH1 = 18, XH2 = 19,  // the pair's second point is the high x1 ghost of V1 / of V2 and V3
           SPECIAL = 20,  // a cell on an x1 face with a divergence-free ghost or the free-surface pressure
           GY_ = 21,      // V1 (+1, +2) has an x2 ghost next to this row
           YS = 24, YT = 25 };  // a cell on an x2 face with a divergence-free ghost / a prescribed normal stress
    unsigned fl = 0;
    {
        const bool in[2] = {in0, in1};
        const bool nrow = !halo && J >= 1 && J <= n2 - 1;
        for (int l = 0; l < 2; ++l) {
            const int xl = x + l;
            fl |= (in[l] ? 1u : 0u) << (IN_ + l);
            fl |= (in[l] && xl < n1 - 1 && y < n2 - 1 ? 1u : 0u) << (E12_ + l);
            fl |= (in[l] && xl < n1 - 1 && y < n2 - 2 ? 1u : 0u) << (E13_ + l);
            fl |= (in[l] && xl < n1 - 2 && y < n2 - 1 ? 1u : 0u) << (E23_ + l);
        }
        for (int f = 0; f < 3; ++f) {
            const int lastI = f == 0 ? n1 - 1 : n1 - 2, lastJ = f == 1 ? n2 - 1 : n2 - 2;
            const bool row = nrow && J <= lastJ;
            const bool lo = MODE == 1 && (o.gmask >> (2 * f) & 1), hi = MODE == 1 && (o.gmask >> (2 * f) & 2);
            const bool a0 = row && (I >= 1 ? I <= lastI : I == 0 && lo);
            const bool a1 = row && I + 1 >= 1 && (I + 1 <= lastI || (I == lastI && hi));
            fl |= (a0 ? 1u : 0u) << (M_ + 2 * f) | (a1 ? 1u : 0u) << (M_ + 2 * f + 1);
            fl |= (row && I + 1 == lastI && hi ? 1u : 0u) << (X_ + f);
            fl |= (row && o.gmask && (J == 1 ? o.gmask >> (6 + 2 * f) & 1 : J == lastJ && (o.gmask >> (7 + 2 * f) & 1)) ? 1u : 0u) << (GY_ + f);
        }
        if (I == 0) fl |= 1u << XLO;
        if (I == n1 - 1) fl |= 1u << XH1;
        if (I == n1 - 2) fl |= 1u << XH2;
        const bool yf = y == 0 || y == n2 - 1;
        if (yin && (p.fs || (o.smask & 3)) && (x <= 0 || x + 1 >= n1 - 1)) fl |= 1u << SPECIAL;
        if (yin && o.smask & (y == 0 ? 4 : (y == n2 - 1 ? 8 : 0))) fl |= 1u << YS;
        if (yin && p.traction && yf) fl |= 1u << YT;
    }
    // whole warps without masks: every cell and edge inside, every node written and no ghost
    const bool wcells = __all_sync(0xffffffffu, (fl & 255u) == 255u);
    constexpr unsigned kStage1Bits = 1u << SPECIAL | 1u << YS | 1u << YT;  // (of no concern to the nodes)
    const bool wnodes = __all_sync(0xffffffffu, ((fl & ~kStage1Bits) >> M_) == 63u);
    auto has = [&](int bit) { return (fl >> bit & 1u) != 0u; };
    // a warp whose two rows lie past the grid (the last tile of a ragged n2) only keeps the barriers: no
    // valid point reads its rows
    const bool busy = halo || y0 + 2 * warp < n2;

    // Spherical: four momentum coefficients wait in shared memory, for registers (spilled ones go to
    // L2, as the shared memory of two blocks leaves almost no L1)
    float2* mom = S.mom[0] + tid;
    constexpr int MS = SW_NT - 32;
    if (G == SPH && !halo) { mom[0] = C.m1_d3; mom[MS] = C.m1_t; mom[2 * MS] = C.m2_d3; mom[3 * MS] = C.m2_n; }
    auto coef = [&](int i, float2 c) { return G == SPH ? const_cast<const float2*>(mom)[i * MS] : c; };

    // ---- carried from plane to plane: input values of plane k for stage 1 of plane k (see the
    // file's head), σ33, DT_R / 2, τ12, τ13, τ23 of plane K-1 for the velocities of plane K
    struct Carry {
        float2 eP, eX, eY, sP, sX, sY;
        float2 s33, dt, t13, t23;
        float t12, u23;
    };
    Carry ca, cb;
    ca.s33 = ca.dt = ca.t13 = ca.t23 = dup(0.f);
    ca.t12 = ca.u23 = 0.f;
    float2 o11, o22, ov1, ov2, ov3;  // σ11, σ22 and the old velocities of this pair at the current plane

    // values of an input tile at row offset db: the pair's points (P) and their x1 neighbours (S)
    auto ldP = [&](const float* A, int db) { return *reinterpret_cast<const float2*>(A + iin + db * SI_X); };
    auto ldS = [&](const float* A, int db, float2 P) { return make_float2(P.y, A[iin + db * SI_X + 2]); };

    // point l of a pair
    auto at = [](float2 v, int l) { return l ? v.y : v.x; };
    auto set = [](float2& v, int l, float q) { v = l ? make_float2(v.x, q) : make_float2(q, v.y); };
    auto rare = [](bool c) { return __builtin_expect(c, 0) != 0; };

    // stresses of plane k from the values n brings along from plane k; leaves those of plane k + 1
    // in m
    auto stage1 = [&](auto par, int k, bool own, const float* A, const float* B, const Carry& n, Carry& m) {
        constexpr int so = decltype(par)::value;  // parity of k - k0: slots
        const float *A2 = A + SI_N, *B2 = B + SI_N, *A3 = A2 + SI_N, *B3 = B2 + SI_N;  // V2, V3 of planes k, k + 1
        auto ld2 = [&](const float* T, int db) { return make_float2(T[iin + db * SI_X + 1], T[iin + db * SI_X + 2]); };
        auto old = [&](const float* T, int f) { return *reinterpret_cast<const float2*>(T + f * SO_N + iold); };
        float2 vP, v11, v22, v33, vdt, v12, v13, v23;
        {
            ov1 = ldP(A, 0); ov2 = ldP(A2, 0); ov3 = ldP(A3, 0);
            float2 a1 = ov1, b1 = ldS(A, 0, a1), a2 = ov2, b2 = ldP(A2, 1), a3 = ov3, b3 = ldP(B3, 0);
            const bool zface = k == 0 || k == n3 - 1;
            if (MODE == 1 && has(YS) && !zface && !has(SPECIAL)) {  // div_ghost<D = 1> of both points
                const bool low = y == 0;
                const float sg = low ? -1.f : 1.f;
                const float2 hh = dup(0.5f), c1 = mul2(C.e1, dup(G == SPH ? 4.f : 2.f)), c2 = add2(C.e2, C.e2);
                const float2 avx = mul2(hh, add2(a1, b1)), vin = low ? b2 : a2;
                const float2 t = fma2(C.a3, sub2(b3, a3), fma2(c1, avx, mul2(vin, fma2(hh, c2, mul2(dup(-sg), C.a2)))));
                const float2 num = mul2(fma2(o.d1, sub2(b1, a1), t), dup(-1.f)), den = fma2(dup(sg), C.a2, mul2(hh, c2));
                const float2 rc = make_float2(rcp_approx(den.x), rcp_approx(den.y)), q = mul2(num, rc);
                const float2 g = fma2(fma2(mul2(den, dup(-1.f)), q, num), rc, q);
                if (low) a2 = g;
                else b2 = g;
            } else if (rare(MODE == 1 && o.smask && (has(SPECIAL) || zface))) {
#pragma unroll 1
                for (int l = 0; l < 2; ++l) {
                    if (!has(IN_ + l)) continue;
                    float w[6] = {at(a1, l), at(b1, l), at(a2, l), at(b2, l), at(a3, l), at(b3, l)};
                    sweep_fill_ghosts<G>(&p, o.smask, x + l, y, k, at(C.a2, l), at(C.a3, l), at(C.e1, l), at(C.e2, l), w);
                    set(a1, l, w[0]); set(b1, l, w[1]); set(a2, l, w[2]); set(b2, l, w[3]); set(a3, l, w[4]); set(b3, l, w[5]);
                }
            }
            const float2 u = mul2(o.d1, sub2(b1, a1)), s1 = add2(a1, b1), e2 = sub2(b2, a2), e3 = sub2(b3, a3);
            float2 div = fma2(C.a3, e3, fma2(C.a2, e2, u));
            float2 D11 = u, D22, D33;
            if (G != CART) {
                const float2 ex = mul2(C.e1, s1);
                D22 = fma2(C.a2, e2, ex);
                if (G == SPH) {
                    const float2 s2 = add2(a2, b2);
                    D33 = fma2(C.e2, s2, fma2(C.a3, e3, ex));
                    div = fma2(C.e2, s2, fma2(C.e1, add2(s1, s1), div));
                } else {
                    D33 = mul2(C.a3, e3);
                    div = fma2(C.e1, s1, div);
                }
                const float2 t = mul2(div, o.third);
                D11 = add2(D11, t); D22 = add2(D22, t); D33 = add2(D33, t);
            } else {
                D22 = mul2(C.a2, e2); D33 = mul2(C.a3, e3);
            }
            const float2 gs = mul2(o.gsc, n.sP), kb = mul2(o.kbc, n.sP);
            const float2 f = div2<LIFT>(n.eP, add2(n.eP, gs), n.sP, o.small);
            const float2 gs2 = add2(gs, gs);
            if (MODE == 1) div = add2(div, old(S.rp[so], 0));
            vP = fma2(mul2(o.nkbc, n.sP), div, old(S.P[so], 0));
            v11 = mul2(fma2(gs2, D11, old(S.tau[so], 0)), f);
            v22 = mul2(fma2(gs2, D22, old(S.tau[so], 1)), f);
            v33 = mul2(fma2(gs2, D33, old(S.tau[so], 2)), f);
            if (has(YT) && !zface) {
                vP = sub2(v22, dup(p.sig2));
            } else if (rare(has(SPECIAL) || (p.traction && zface))) {
#pragma unroll 1
                for (int l = 0; l < 2; ++l) {
                    if (!has(IN_ + l)) continue;
                    float P = at(vP, l);
                    if (p.traction) traction_pressure(y, k, n2, n3, at(v22, l), at(v33, l), p.sig2, p.sig3, P);
                    if (p.fs && x + l == n1 - 1)
                        P = at(v11, l) + (MODE == 1 ? 0.f : p.top_load[x + l + d.sy * y + d.sz * k]) + p.fs_kappa * (0.5f * at(s1, l));
                    set(vP, l, P);
                }
            }
            vdt = div2<LIFT>(o.vp, fma2(gs, f, kb), n.sP, o.small);
        }
        float2 st = dup(0.f);  // LIFT: ηSM of the cell that all three edges have in common
        auto sums = [&](const float* A, float2& P, float2& X0, float2& X, float2& Y) {
            P = ldP(A, 0);
            const float2 s = ldS(A, 0, P), q = ldP(A, 1), t = ldS(A, 1, q);
            X0 = add2(P, s); X = add2(q, t); Y = add2(s, t);
            if (LIFT) st = t;
        };
        float2 eX0, sX0;
        sums(B + 3 * SI_N, m.eP, eX0, m.eX, m.eY);
        sums(B + 4 * SI_N, m.sP, sX0, m.sX, m.sY);
        // edge update from the sums s4, e4 of ηSM and η over four cells, aG = GSDT s4 / 4, aE = e4 / 4:
        // (τ + aG D) aE / (aE + aG) with D4 = D / 4
        auto edge = [&](float2 told, float2 s4, float2 e4, float2 D4) {
            const float2 g4 = mul2(o.gsc, s4);
            return mul2(fma2(g4, D4, told), div2<LIFT>(e4, add2(e4, g4), st, o.small));
        };
        const float2 b1T = ld2(B, 1), b2T = ld2(B2, 1), b3Q = ldP(B3, 1), b3T = ldS(B3, 1, b3Q);
        {
            const float2 b1S = ld2(B, 0), b2Q = ldP(B2, 1);
            float2 D = fma2(C.e12_d2, sub2(b1T, b1S), mul2(o.d1q, sub2(b2T, b2Q)));
            if (G != CART) D = fma2(C.e12_h, add2(b2Q, b2T), D);
            v12 = edge(old(S.tau[so], 3), add2(sX0, m.sX), add2(eX0, m.eX), D);
        }
        {
            float2 D = fma2(C.e13_d3, sub2(b1T, ld2(A, 1)), mul2(o.d1q, sub2(b3T, b3Q)));
            if (G == SPH) D = fma2(C.e12_h, add2(b3Q, b3T), D);
            v13 = edge(old(S.tau[so], 4), add2(n.sX, m.sX), add2(n.eX, m.eX), D);
        }
        {
            const float2 b3S = ld2(B3, 0);
            float2 D = fma2(C.e23_d3, sub2(b2T, ld2(A2, 1)), mul2(C.e23_d2, sub2(b3T, b3S)));
            if (G == SPH) D = fma2(C.e23_h, add2(b3S, b3T), D);
            v23 = edge(old(S.tau[so], 5), add2(n.sY, m.sY), add2(n.eY, m.eY), D);
        }

        const bool k12 = k < n3 - 2, k1x = k < n3 - 1;
        const unsigned gb = 4u * (unsigned)(gxy + d.sz * k);  // byte offset (owned points only: >= 0)
        float2 o33 = sub2(v33, vP);
        o11 = sub2(v11, vP); o22 = sub2(v22, vP);
        if (!(wcells && k12)) {  // zero outside the grid (a pair's first point is inside where its second is)
            const bool i0 = has(IN_), i1 = has(IN_ + 1);
            vP = keep2(vP, i0, i1); v11 = keep2(v11, i0, i1); v22 = keep2(v22, i0, i1); v33 = keep2(v33, i0, i1);
            o11 = keep2(o11, i0, i1); o22 = keep2(o22, i0, i1); o33 = keep2(o33, i0, i1); vdt = keep2(vdt, i0, i1);
            v12 = keep2(v12, has(E12_) && k12, has(E12_ + 1) && k12);
            v13 = keep2(v13, has(E13_) && k1x, has(E13_ + 1) && k1x);
            v23 = keep2(v23, has(E23_) && k1x, has(E23_ + 1) && k1x);
        }
        if (own && has(IN_)) {  // (zeros where the second point, or an edge of the first, is padding)
            st_pair(o.P, gb, vP); st_pair(o.t11, gb, v11); st_pair(o.t22, gb, v22); st_pair(o.t33, gb, v33);
            st_pair(o.t12, gb, v12); st_pair(o.t13, gb, v13); st_pair(o.t23, gb, v23);
        }
        m.s33 = o33; m.dt = vdt; m.t12 = v12.x; m.u23 = v23.x;
        auto put = [&](float* W, float2 v) { *reinterpret_cast<float2*>(W + ist) = v; };
        if (halo && lane == 31) return;
        put(S.q[0], o11); put(S.q[1], o22); put(S.q[2], o33); put(S.q[3], vdt);
        put(S.e[so][0], v12); put(S.e[so][1], v13); put(S.e[so][2], v23);
    };

    // velocities of plane K at the nodes (I, J), (I + 1, J) from the stresses of planes K-1 and K
    // (n, m: what stage 1 of plane K took and left)
    auto velocity = [&](auto par, int K, bool own, const Carry& n, Carry& m) {
        constexpr int so = decltype(par)::value;
        const float *E12p = S.e[1 - so][0] + ist, *E13p = S.e[1 - so][1] + ist, *E23p = S.e[1 - so][2] + ist;
        const float *E13 = S.e[so][1] + ist - SR_X, *E23 = S.e[so][2] + ist - SR_X;
        const float2 c13 = make_float2(E13[-1], E13[0]), c23 = make_float2(E23[-1], E23[0]);
        m.t13 = c13; m.t23 = c23;
        const float2 p13 = n.t13, p23 = n.t23, o33 = m.s33, odt = m.dt;
        if (own && K >= 1 && K <= n3 - 1) {
            const unsigned gb = 4u * (unsigned)(gxy + d.sz * K);  // byte offset (valid nodes only: >= 0)
            const float2 b12 = *reinterpret_cast<const float2*>(E12p - SR_X);               // τ12 (I, J-1, K-1)
            const float2 t12a = make_float2(E12p[-1], n.t12), t12b = make_float2(E12p[-SR_X - 1], b12.x);
            const float *Q11 = S.q[0] + ist, *Q22 = S.q[1] + ist, *Q33 = S.q[2] + ist, *QDT = S.q[3] + ist;
            const float* R = MODE == 1 ? S.rv[so] + (b - 1) * SWX + (a - 1) : S.rp[so] + iold;
            auto rv = [&](int f) { return *reinterpret_cast<const float2*>(R + f * SV_N); };
            const float2 gh = dup(-0.5f * p.g), rc = MODE == 0 ? rv(0) : dup(0.f);
            float2 u1, u2, u3;
            {  // V1 (I-1/2, J, K), cell m = (I-1, J, K)
                const float2 m11 = make_float2(Q11[-1], o11.x);
                float2 r1 = fma2(coef(0, C.m1_d3), sub2(c13, p13), mul2(o.d1, sub2(o11, m11)));
                float2 t = mul2(o.d2, sub2(t12a, t12b));  // terms with the factor 1/x1
                if (G != CART) {
                    const float2 m22 = add2(make_float2(Q22[-1], o22.x), o22);
                    if (G == SPH) {
                        const float2 m33 = add2(make_float2(Q33[-1], o33.x), o33);
                        t = add2(t, fma2(o.half, add2(m22, m33), add2(m11, o11)));
                        r1 = fma2(coef(1, C.m1_t), add2(t12a, t12b), r1);
                    } else {
                        t = fma2(o.half, sub2(m22, add2(m11, o11)), t);
                    }
                    r1 = fma2(C.m1_i, t, r1);
                } else {
                    r1 = add2(r1, t);
                }
                if (MODE == 1) r1 = add2(r1, rv(0));
                else if (G != CART) r1 = fma2(gh, add2(make_float2(R[-1], rc.x), rc), r1);
                u1 = fma2(r1, add2(make_float2(QDT[-1], odt.x), odt), ov1);
            }
            {  // V2 (I, J-1/2, K), cell m = (I, J-1, K)
                const float2 m22 = *reinterpret_cast<const float2*>(Q22 - SR_X);
                float2 r2 = fma2(coef(2, C.m2_d3), sub2(c23, p23), fma2(C.a2, sub2(o22, m22), mul2(o.d1, sub2(b12, t12b))));
                if (G != CART) r2 = fma2(C.m2_s, add2(b12, t12b), r2);
                if (G == SPH) {
                    const float2 m33 = *reinterpret_cast<const float2*>(Q33 - SR_X);
                    r2 = fma2(coef(3, C.m2_n), sub2(add2(m22, o22), add2(m33, o33)), r2);
                }
                if (MODE == 1) r2 = add2(r2, rv(1));
                u2 = fma2(r2, add2(*reinterpret_cast<const float2*>(QDT - SR_X), odt), ov2);
            }
            {  // V3 (I, J, K-1/2), cell m = (I, J, K-1)
                const float2 t13a = *reinterpret_cast<const float2*>(E13p - SR_X), t23a = make_float2(E23p[-1], n.u23);
                float2 r3 = fma2(C.a3, sub2(o33, n.s33), fma2(C.a2, sub2(t23a, p23), mul2(o.d1, sub2(t13a, p13))));
                if (G == SPH) {
                    const float2 t = add2(t23a, p23);
                    r3 = fma2(C.m2_s, add2(t13a, p13), fma2(C.e2, add2(t, t), r3));
                }
                if (G == CYL) r3 = fma2(C.e1, add2(t13a, p13), r3);
                if (MODE == 1) {
                    r3 = add2(r3, rv(2));
                } else if (G == CART) {  // ρ of plane K-1: its slot is being refilled
                    const float2 rm = make_float2(has(M_ + 4) ? p.rho[gxy + d.sz * (K - 1)] : 0.f, has(M_ + 5) ? p.rho[gxy + d.sz * (K - 1) + 1] : 0.f);
                    r3 = fma2(gh, add2(rm, rc), r3);
                }
                u3 = fma2(r3, add2(n.dt, odt), ov3);
            }
            if (wnodes && K > 1 && K <= n3 - 3) {
                st_pair(o.V1, gb, u1); st_pair(o.V2, gb, u2); st_pair(o.V3, gb, u3);
                return;
            }
            // Nodes next to the grid's faces, with MODE 1 also their ghosts: on x1 within the pair (then still one
            // store) or after it, on x2 and x3 the same once more at the face's offset, edges and corners
            // included.  The lanes of a warp stay together here: only the extra stores are masked.
            auto put = [&](float* A, int f, float2 v, int high, int lastK) {
                if (MODE == 1) {
                    if (has(XLO)) v.x = o.gf[f] * v.y;
                    if (has(high)) v.y = o.gf[f] * v.x;
                }
                auto row = [&](unsigned at, float2 w) {
                    st_pair(A, at, w, has(M_ + 2 * f), has(M_ + 2 * f + 1));
                    if (MODE == 1 && has(X_ + f)) st_at(A, at + 8u, o.gf[f] * w.y);
                };
                row(gb, v);
                if (MODE == 0) return;
                const bool gy = has(GY_ + f);
                const bool gz = K == 1 ? (o.gmask >> (12 + 2 * f) & 1) : K == lastK && (o.gmask >> (13 + 2 * f) & 1);
                const unsigned oy = (unsigned)(J == 1 ? -4 * d.sy : 4 * d.sy), oz = (unsigned)(K == 1 ? -4 * d.sz : 4 * d.sz);
                const float2 vy = mul2(v, dup(o.gf[3 + f]));
                if (gy) row(gb + oy, vy);
                if (gz) {
                    row(gb + oz, mul2(v, dup(o.gf[6 + f])));
                    if (gy) row(gb + oy + oz, mul2(vy, dup(o.gf[6 + f])));
                }
            };
            if (K <= n3 - 2) {
                put(o.V1, 0, u1, XH1, n3 - 2);
                put(o.V2, 1, u2, XH2, n3 - 2);
            }
            put(o.V3, 2, u3, XH2, n3 - 1);
        }
    };

    // ---- the march
    if (halo) ok = mbar_wait(&S.bar_0, 0u);
    __syncthreads();
    {  // carried values of plane k0
        auto sums = [&](const float* A, float2& P, float2& X, float2& Y) {
            P = ldP(A, 0);
            const float2 s = ldS(A, 0, P), q = ldP(A, 1), t = ldS(A, 1, q);
            X = add2(q, t); Y = add2(s, t);
        };
        sums(S.in[0] + 3 * SI_N, ca.eP, ca.eX, ca.eY);
        sums(S.in[0] + 4 * SI_N, ca.sP, ca.sX, ca.sY);
    }

    // one plane: waits, stage 1, copies of the planes after, velocities
    const float *A = S.in[0], *B = S.in[1];  // input planes K, K + 1
    auto step = [&](auto par, int K, const Carry& n, Carry& m) {
        constexpr int so = decltype(par)::value;
        const bool own = K >= kA;
        if (halo) wait(&S.bar_s[so], so);
        __syncthreads();  // copies have landed; the velocities of plane K-1 are done with the shared stresses
        if (busy) stage1(par, K, own && !halo, A, B, n, m);
        if (halo && own) wait(&S.bar_v[so], 2 + so);
        __syncthreads();
        if (!halo) {
            if (busy) velocity(par, K, own, n, m);
        } else if (issuer && ok) {
            if (K + 2 < kB) issue_stage(K + 2);
            if (own && K + 1 < kB) issue_rhs(K + 1);
        }
        A = B;
        B = B == S.in[2] ? S.in[0] : B + 5 * SI_N;
    };
    for (int K = k0; K < kB; K += 2) {  // two planes a turn, so that the carried pairs need no moves
        step(std::integral_constant<int, 0>{}, K, ca, cb);
        if (K + 1 >= kB) break;
        step(std::integral_constant<int, 1>{}, K + 1, cb, ca);
        // The next grid's blocks may come once every block is within two planes of its end: their set-up then fills the
        // tail of this grid.  us per sweep, released at the end (implicitly) and so: 63^3 12.9 and 11.8, 131 x 117 x 101
        // 45.2 and 44.6, 255^3 305.2 and 304.6, sector 28 x 29 x 158 10.6 and 9.3; at the start of the block 28 x 75 x 72 became
        // 11.6 (10.6; so 10.1), as early blocks leave the SMs unevenly filled.
        if (K + 4 >= kB) asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    }
    // Without a time-out every issued copy has been waited for, so none is in flight when the
    // block exits.  After a time-out copies issued before it may still be landing in this
    // block's shared memory as it exits and the state it wrote is suspect: the host reads the
    // flag after the launch and treats it as fatal for the context.
    if (halo && !ok && err) atomicExch(err, 1);
}

template <int G, int MODE, bool LIFT>
__global__ void __launch_bounds__(SW_NT, 2) k_sweep(const __grid_constant__ KP<float> p, const __grid_constant__ SweepOut<float> o, int kchunk,
                                                    const __grid_constant__ SweepMaps maps, int* __restrict__ err) {
    sweep_body<G, MODE, LIFT>(p, o, kchunk, maps.m, err, blockIdx.x, blockIdx.y, blockIdx.z);
}

}  // namespace sph
