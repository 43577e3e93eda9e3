// Arithmetic of the FP64 kernels in few FP64 instructions.
//
// GB300 executes about two FP64 operations per SM and clock (1/64 of its FP32 rate), so
// the FP64 path is bound by the number of FP64 instructions and hardly by anything else.
#pragma once
#include <cmath>

#include "sph_core.cuh"

namespace sph {

// a / b in five FP64 operations, for operands of 2^-500 .. 2^500 in magnitude (quotient and residuals are then inside the
// range of normal numbers): PTX's approximate reciprocal r (relative error e near 2^-20), one Newton step (e^2), the
// quotient a r and one step by its residual, q += r (a - b q) (Markstein, IBM J. Res. Dev. 34, 1990), which leaves e^4
// before the last rounding: the IEEE quotient but for about one pair of operands in 2^24.  (Two residual steps with
// the reciprocal as it comes take as many operations and leave e^3: 297 of 2^20 quotients were one unit off.)
__device__ __forceinline__ double mid_div(double a, double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    r = fma(fma(-b, r, 1.0), r, r);
    const double q = a * r;
    return fma(fma(-b, q, a), r, q);
}
__device__ __forceinline__ float mid_div(float a, float b) { return pdiv(a, b); }

// whether every number added is positive and of 2^-E .. 2^E (integer operations, no FP64 issue)
template <typename T, int E>
struct MidRange {
    unsigned lo = ~0u, hi = 0u;
    __device__ __forceinline__ void add(T x) {
        if constexpr (sizeof(T) == 8) {
            const unsigned v = (unsigned)__double2hiint(x);
            lo = min(lo, v);
            hi = max(hi, v);
        }
    }
    __device__ __forceinline__ bool ok() const { return sizeof(T) != 8 || (lo >= (1023u - E) << 20 && hi < (1023u + E) << 20); }
};

// a / b of any operands: those that are not positive or outside the range, infinities and NaN among them, by the IEEE division
__device__ __forceinline__ double near_div(double a, double b) {
    MidRange<double, 500> m;
    m.add(a);
    m.add(b);
    return m.ok() ? mid_div(a, b) : a / b;
}

// square root of a positive normal x in seven FP64 operations: the approximate reciprocal root, one
// coupled (Goldschmidt) step for the root and half its reciprocal, and the residual correction; others by sqrt()
__device__ __forceinline__ double mid_sqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double g = x * y, h = 0.5 * y;
    const double e = fma(-g, h, 0.5);
    const double g1 = fma(g, e, g);
    return fma(fma(-g1, g1, x), fma(h, e, h), g1);
}
__device__ __forceinline__ double fast_sqrt(double x) { return (unsigned)__double2hiint(x) - 0x00200000u < 0x7fc00000u ? mid_sqrt(x) : sqrt(x); }

// ---------------------------------------------------------------------------
// x^c of positive normal numbers, after the table-driven scheme of P. T. P. Tang (ACM TOMS 15-18, 1989-1992):
// log2 x = E + log2(1/C_i) + log2(1 + r), r = m C_i - 1 with C_i ~ 1/m of the interval of m's leading seven
// bits, as an exact head and a short tail; c log2 x the same way; 2^y = 2^n 2^(j/64) 2^g.  About 24 FP64
// operations and an error below 1.1 units in the last place while |c log2 x| < 1000, against some hundred
// operations of pow().  The tables are made on the host (fill_pow_tables).
constexpr int kLogN = 128, kExpN = 64;
constexpr int kPowTab = 3 * kLogN + kExpN;  // doubles: C_i, head, tail of log2(1/C_i); 2^(j/64)

__device__ __forceinline__ bool normal_pos(double x) { return (unsigned)__double2hiint(x) - 0x00100000u < 0x7fe00000u; }

// log2 of a positive normal x: head (a multiple of 2^-40: sums of a few heads are exact) and tail
__device__ __forceinline__ void log2_parts(const double* __restrict__ tab, double x, double& head, double& tail) {
    const int hi = __double2hiint(x);
    const int i = (hi >> 13) & (kLogN - 1);
    const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(x));
    const double r = fma(m, __ldg(tab + i), -1.0);  // |r| < 2^-8
    // log2(1 + r) = sum (-1)^(k+1) r^k / (k ln 2), to r^6: the next term is below 2^-58
    double p = -0.2404491734814939;
    p = fma(p, r, 0.28853900817779266);
    p = fma(p, r, -0.36067376022224085);
    p = fma(p, r, 0.4808983469629878);
    p = fma(p, r, -0.7213475204444817);
    p = fma(p, r, 1.4426950408889634);
    tail = fma(p, r, __ldg(tab + 2 * kLogN + i));
    head = (double)((hi >> 20) - 1023) + __ldg(tab + kLogN + i);
}
// 2^(y + t), |y| < 1000, t a small correction
__device__ __forceinline__ double exp2_parts(const double* __restrict__ tab, double y, double t) {
    const double big = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer in the low word
    const double s = fma(y, (double)kExpN, big);
    const int n = __double2loint(s);
    const double g = fma(s - big, -1.0 / kExpN, y) + t;  // |g| <= 2^-7
    // 2^g - 1 = sum (g ln 2)^k / k!, to g^6: the next term is below 2^-66
    double p = 0.0001540353039338161;
    p = fma(p, g, 0.0013333558146428443);
    p = fma(p, g, 0.009618129107628477);
    p = fma(p, g, 0.05550410866482158);
    p = fma(p, g, 0.24022650695910072);
    p = fma(p, g, 0.6931471805599453);
    const double T = __ldg(tab + 3 * kLogN + (n & (kExpN - 1)));
    const double v = fma(T * g, p, T);
    return __hiloint2double(__double2hiint(v) + ((n >> 6) << 20), __double2loint(v));
}
__device__ __forceinline__ double fast_pow(const double* __restrict__ tab, double x, double c) {
    if (normal_pos(x)) {
        double h, t;
        log2_parts(tab, x, h, t);
        const double y = c * h;
        if ((__double2hiint(y) & 0x7fffffff) < 0x408f4000)  // |y| < 1000
            return exp2_parts(tab, y, fma(c, t, fma(c, h, -y)));
    }
    return pow(x, c);
}

// x^m for small m >= 0, from x^2 = s: m / 2 factors s and one x where m is odd
__device__ __forceinline__ double small_pow(double x, double s, int m) {
    if (m <= 0) return 1.0;
    if (m == 1) return x;
    const double s2 = s * s;
    double v = m & 2 ? s : 1.0;
    if (m & 4) v = m & 2 ? v * s2 : s2;
    if (m & 8) v = m & 6 ? v * (s2 * s2) : s2 * s2;
    return m & 1 ? v * x : v;
}

// x^(p/q), p = 1, 2, 3, q = 3, 4, 5, 8, of x with an exponent below 300 in magnitude: a start y from FP32 logarithm
// and exponential (relative error below 1e-6; the exponent of x is split off, so also far from 1) and one step of
// Halley's method (p / q = e + el), y += y (rho - 1) (z - y^q) / (rho y^q + z), z = x^p, rho = (q + 1) / (q - 1), which
// cubes the error.  10 - 13 FP64 operations, table-driven power 24.  Largest error over 2^18 arguments in 2^-295 .. 2^295:
// 1.7e-16 (table: 2.1e-16, and 5e-15 where p/q is not a double).
__device__ __forceinline__ double root_pow(double x, int p, int q, double rho, float e, float el) {
    const int hi = __double2hiint(x);
    const float E = (float)((hi >> 20) - 1023);
    const float m = __int_as_float(0x3f800000 | ((hi & 0x000fffff) << 3) | (int)((unsigned)__double2loint(x) >> 29));
    float l, y32;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(m));
    const float h = e * E, n = rintf(h);
    const float f = (h - n) + fmaf(e, l, fmaf(el, E, fmaf(e, E, -h)));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y32) : "f"(f));
    const int b = __float_as_int(y32);  // to double with 2^n, by integer operations
    const double y = __hiloint2double((b >> 3) + ((1023 - 127 + (int)n) << 20), b << 29);
    const double y2 = y * y;
    double a = q == 3 ? y2 * y : y2 * y2;
    if (q == 5) a *= y;
    if (q == 8) a *= a;
    double z = x;
    if (p >= 2) z *= x;
    if (p == 3) z *= x;
    const double den = fma(rho, a, z), num = z - a;
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(den));
    const double d = num * r;
    return fma(y * (rho - 1.0), fma(fma(-den, d, num), r, d), y);
}
__device__ __forceinline__ bool root_range(double x) { return (unsigned)__double2hiint(x) - 0x2d300000u < 0x25800000u; }  // 2^-300 .. 2^300

inline void fill_pow_tables(double* tab) {
    for (int i = 0; i < kLogN; ++i) {
        const double C = (double)(float)(1.0 / (1.0 + (i + 0.5) / kLogN));
        const long double L = -std::log2((long double)C), u = 1099511627776.0L;  // 2^40
        const double head = (double)(std::nearbyint(L * u) / u);
        tab[i] = C;
        tab[kLogN + i] = head;
        tab[2 * kLogN + i] = (double)(L - (long double)head);
    }
    for (int j = 0; j < kExpN; ++j) tab[3 * kLogN + j] = (double)std::exp2((long double)j / kExpN);
}

}  // namespace sph
