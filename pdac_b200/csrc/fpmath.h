// fpmath.h -- exp and pow in IEEE binary64 arithmetic that give the same
// bits on the host and on the device.
//
// The per-step path raises to real powers in the drag law (drag.f:60-157),
// the gas-particle heat transfer (hvs.f:9-83), the collision integral of
// the gas viscosity (visc.f:37-148, with exp), the particle repulsion
// (tilde.f:362-416) and the sub-grid filter (turbo.f).  The C library and
// CUDA's math library may round these last bits differently, and one last
// bit is enough to put a corrector cell whose |dg| lies within a rounding
// error of conv on the other side of the convergence test, after which two
// runs differ at the level of delg.  The routines below use only +, -, *, /,
// fma, rint and ldexp -- each exactly specified by IEEE 754, so the same on
// the host (C++, no FMA contraction) and the device (CUDA, -fmad=false) --
// and tables written out as hexadecimal literals (fpmath_tables.h, made by
// gen_fpmath_tables.py).  The engine's kernels and the CPU oracle both call
// them, so both compute the same bits.
//
// Methods: P. T. P. Tang, "Table-driven implementation of the exponential
// function in IEEE floating-point arithmetic", ACM TOMS 15 (1989) 144-157
// (exp = 2^m * 2^(j/32) * exp(r), |r| <= ln2/64), and "Table-driven
// implementation of the logarithm function in IEEE floating-point
// arithmetic", ACM TOMS 16 (1990) 378-400 (log x = m ln2 + log F +
// log1p(f/F), F = 1 + j/128).  pow(x, y) = exp(y log x) with log x carried
// as a double-double and y log x formed with fma, so the result is within
// about one unit in the last place (tests/test_fpmath.py checks it against
// the C library over the ranges the path uses).
#pragma once
#include <cmath>
#include <cstring>
#include <limits>

#include "fpmath_tables.h"

#ifdef __CUDACC__
#define PDAC_FP_FN __host__ __device__ __forceinline__
#else
#define PDAC_FP_FN inline
#endif

namespace pdac_fp {

// a / b for a divisor used many times: with y = RN(1 / b) computed once by an
// IEEE division, the quotient RN(a / b) from two corrections of a y by its
// exactly computed residual (P. W. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34
// (1990) 111-119: when q is within one ulp of a / b and y is the correctly
// rounded reciprocal, RN(q + y RN(a - b q)) is RN(a / b)).  The first
// correction brings a y, which may be two ulps off, within one; the second is
// the theorem's.  It holds away from the ends of the exponent range: outside
// the ranges tested below the quotient is divided, so the result is the
// division's for every a and b.  A chain of five 8.8-cycle operations on the
// device instead of a 127-cycle division.
struct Recip {
    double b, y;
};
PDAC_FP_FN Recip recip(double b) {
    const double m = fabs(b);
    return {b, m > 1e-30 && m < 1e30 ? 1.0 / b : std::numeric_limits<double>::quiet_NaN()};
}
PDAC_FP_FN double div_by(double a, const Recip &R) {
    double q = a * R.y;
    q = fma(fma(-R.b, q, a), R.y, q);
    q = fma(fma(-R.b, q, a), R.y, q);
    const double m = fabs(a);
    if (!(m > 1e-250 && m < 1e250) || q != q) q = a / R.b;
    return q;
}

// |(a - b) / a| <= tol, the relative-change test of a fixed-point iteration,
// decided without the division unless the quotient lies within 1e-14 of tol
// (1e-14 covers the rounding of every operation here many times over)
PDAC_FP_FN bool rel_change_within(double a, double b, double tol) {
    const double d = fabs(a - b), m = fabs(a), t = m * tol;
    if (m > 1e-250 && m < 1e250) {
        if (d <= t * (1.0 - 1e-14)) return true;
        if (d >= t * (1.0 + 1e-14)) return false;
    }
    return fabs((a - b) / a) <= tol;
}

#ifdef __CUDACC__
__constant__ const double kExp2Tab[64] = PDAC_EXP2_TABLE;
__constant__ const double kLogTab[258] = PDAC_LOG_TABLE;
__constant__ const double kInvFTab[129] = PDAC_LOG_INVF_TABLE;
#endif
static const double hExp2Tab[64] = PDAC_EXP2_TABLE;
static const double hLogTab[258] = PDAC_LOG_TABLE;
static const double hInvFTab[129] = PDAC_LOG_INVF_TABLE;

PDAC_FP_FN double exp2_tab(int q) {
#ifdef __CUDA_ARCH__
    return kExp2Tab[q];
#else
    return hExp2Tab[q];
#endif
}
PDAC_FP_FN double log_tab(int q) {
#ifdef __CUDA_ARCH__
    return kLogTab[q];
#else
    return hLogTab[q];
#endif
}
PDAC_FP_FN double invf_tab(int q) {
#ifdef __CUDA_ARCH__
    return kInvFTab[q];
#else
    return hInvFTab[q];
#endif
}

PDAC_FP_FN double fma_(double a, double b, double c) {
#ifdef __CUDA_ARCH__
    return __fma_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}
PDAC_FP_FN double rint_(double x) {
#ifdef __CUDA_ARCH__
    return rint(x);
#else
    return std::nearbyint(x);
#endif
}
PDAC_FP_FN double ldexp_(double x, int e) {
#ifdef __CUDA_ARCH__
    return ldexp(x, e);
#else
    return std::ldexp(x, e);
#endif
}
PDAC_FP_FN double frexp_(double x, int *e) {
#ifdef __CUDA_ARCH__
    return frexp(x, e);
#else
    return std::frexp(x, e);
#endif
}

// v 2^m, as ldexp: where the result is normal the product with the power of
// two, whose bits are m + 1023 in the exponent field, is exact (v in [1/2, 4))
PDAC_FP_FN double scale2(double v, int m) {
    if (m < -1020 || m > 1020) return ldexp_(v, m);
    const unsigned long long b = (unsigned long long)(m + 1023) << 52;
    double p;
#ifdef __CUDA_ARCH__
    p = __longlong_as_double((long long)b);
#else
    std::memcpy(&p, &b, 8);
#endif
    return v * p;
}
// x = 2^e y with y in [1, 2), for finite x > 0
PDAC_FP_FN double split2(double x, int &e) {
    unsigned long long b;
#ifdef __CUDA_ARCH__
    b = (unsigned long long)__double_as_longlong(x);
#else
    std::memcpy(&b, &x, 8);
#endif
    const int f = (int)(b >> 52);
    if (f == 0) {  // subnormal
        const double y = frexp_(x, &e);
        e = e - 1;
        return y * 2.0;
    }
    e = f - 1023;
    b = (b & 0x000fffffffffffffull) | 0x3ff0000000000000ull;
    double y;
#ifdef __CUDA_ARCH__
    y = __longlong_as_double((long long)b);
#else
    std::memcpy(&y, &b, 8);
#endif
    return y;
}

// exp(zh + zl) for |zl| no larger than an ulp or so of zh
PDAC_FP_FN double exp_dd(double zh, double zl) {
    if (zh != zh) return zh;
    if (zh > 709.782712893384) return std::numeric_limits<double>::infinity();
    if (zh < -745.2) return 0.0;
    const double N = rint_(zh * PDAC_INV_LN2_32);
    const int n = (int)N, j = n & 31, m = (n - j) / 32;
    double r = fma_(-N, PDAC_LN2_32_HI, zh);
    r = fma_(-N, PDAC_LN2_32_LO, r) + zl;
    // exp(r) - 1 to degree 6; |r| <= ln2/64, so the first term left out is
    // below 4e-18 of the result
    const double q = r * r * (0x1.0p-1 + r * (0x1.5555555555555p-3 + r * (0x1.5555555555555p-5 +
                                                                     r * (0x1.1111111111111p-7 +
                                                                          r * 0x1.6c16c16c16c17p-10))));
    const double p = r + q;
    const double th = exp2_tab(2 * j), tl = exp2_tab(2 * j + 1);
    const double s = th + tl;
    return scale2(th + (tl + s * p), m);
}

PDAC_FP_FN double exp(double x) { return exp_dd(x, 0.0); }

// log x as hi + lo, for finite x > 0
PDAC_FP_FN void log_dd(double x, double &hi, double &lo) {
    int e;
    const double y = split2(x, e);
    int j = (int)rint_((y - 1.0) * 128.0);
    j = j < 0 ? 0 : (j > 128 ? 128 : j);  // y in [1, 2) gives 0 .. 128; the table has 129 entries
    const double F = 1.0 + (double)j * 0x1.0p-7;
    const double f = y - F;                    // exact: |f| <= 1/256
    // f/F = g + gl: both quotients by the tabulated 1/F as in div_by (f is 0 or
    // a multiple of 2^-52, so no operand comes near the ends of the range)
    const double iF = invf_tab(j);
    double g = f * iF;
    g = fma_(fma_(-F, g, f), iF, g);
    g = fma_(fma_(-F, g, f), iF, g);
    const double d = fma_(-g, F, f);
    double gl = d * iF;
    gl = fma_(fma_(-F, gl, d), iF, gl);
    gl = fma_(fma_(-F, gl, d), iF, gl);
    // log1p(g) - g to degree 6 in g; |g| <= 1/256, the first term left out is
    // below 3e-18
    const double poly = g * g * (-0x1.0p-1 + g * (0x1.5555555555555p-2 + g * (-0x1.0p-2 + g * (0x1.999999999999ap-3 +
                                                                                       g * -0x1.5555555555555p-3))));
    const double a = (double)e * PDAC_LN2_HI;  // exact: the table's ln2 keeps 42 significant bits
    const double b = log_tab(2 * j);
    // two exact sums (Knuth's TwoSum), then the small parts
    double s1 = a + b, bb = s1 - a, t1 = (a - (s1 - bb)) + (b - bb);
    double s2 = s1 + g;
    bb = s2 - s1;
    double t2 = (s1 - (s2 - bb)) + (g - bb);
    double l = t1 + t2 + ((double)e * PDAC_LN2_LO + log_tab(2 * j + 1) + gl + poly);
    hi = s2 + l;
    lo = l - (hi - s2);
}

// x^y for the path's arguments: x >= 0 (x < 0 gives NaN unless y is an
// integer), with the IEEE special cases the path can meet.  Written without
// recursion: a recursive device function leaves the kernel's stack size to
// the runtime's default limit instead of the size the compiler computes.
PDAC_FP_FN double pow(double x, double y) {
    if (y == 0.0 || x == 1.0) return 1.0;
    if (x != x || y != y) return x + y;
    bool negate = false;
    if (x < 0.0) {
        if (y != rint_(y)) return std::numeric_limits<double>::quiet_NaN();
        negate = rint_(y * 0.5) * 2.0 != y;  // an odd integer power keeps the sign
        x = -x;
    }
    double r;
    if (x == 0.0) r = y > 0.0 ? 0.0 : std::numeric_limits<double>::infinity();
    else if (x == std::numeric_limits<double>::infinity()) r = y > 0.0 ? x : 0.0;
    else {
        double lh, ll;
        log_dd(x, lh, ll);
        const double zh = y * lh;
        const double zl = fma_(y, lh, -zh) + y * ll;
        r = exp_dd(zh, zl);
    }
    return negate ? -r : r;
}

// pow of one base to several exponents: its logarithm once.  y finite, not 0
// and not an integer.
struct PowOf {
    double x, lh, ll;
    bool plain;
};
PDAC_FP_FN PowOf pow_of(double x) {
    PowOf b = {x, 0.0, 0.0, x > 0.0 && x < std::numeric_limits<double>::infinity() && x != 1.0};
    if (b.plain) log_dd(x, b.lh, b.ll);
    return b;
}
PDAC_FP_FN double pow_log(double lh, double ll, double y) {
    const double zh = y * lh;
    return exp_dd(zh, fma_(y, lh, -zh) + y * ll);
}
PDAC_FP_FN double pow(const PowOf &b, double y) {
    if (b.plain) return pow_log(b.lh, b.ll, y);
    if (b.x == 1.0) return 1.0;
    if (b.x != b.x) return b.x + y;
    if (b.x < 0.0) return std::numeric_limits<double>::quiet_NaN();
    if (b.x == 0.0) return y > 0.0 ? 0.0 : std::numeric_limits<double>::infinity();
    return y > 0.0 ? b.x : 0.0;
}

// pow(10, y): log 10 as log_dd(10) gives it
#define PDAC_LOGDD_10_HI 0x1.26bb1bbb55516p+1
#define PDAC_LOGDD_10_LO -0x1.f48ad494ea4p-53
PDAC_FP_FN double pow10(double y) { return pow_log(PDAC_LOGDD_10_HI, PDAC_LOGDD_10_LO, y); }

}  // namespace pdac_fp
