"""div_by and rel_change_within of pdac_b200/csrc/fpmath.h against the
division they stand for: the same bits, the same decisions, for operands over
the whole exponent range, exact and near-halfway quotients and the IEEE
special values.  The reciprocal-based quotient is correctly rounded, so no
tolerance is involved."""
import ctypes as C
import os
import subprocess

import pytest

SRC = r"""
#include <cstdint>
#include <cstring>
#include "fpmath.h"
static uint64_t s;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double val(int kind) {
    static const double special[] = {0.0, -0.0, 1.0, -1.0, INFINITY, -INFINITY, NAN, 5e-324, -5e-324, 2.2e-308, 1e-250,
                                     1e250, 1e-251, 1e251, 1e-30, 1e30, 1.7e308, 0.018, 0.02896442, 8.31432};
    if (kind == 0) return special[rnd() % 20];
    uint64_t m = rnd() & 0xfffffffffffffull, sg = rnd() & 0x8000000000000000ull, e;
    if (rnd() % 4 == 0) m &= ~0ull << (rnd() % 52);              // short significands: exact and halfway quotients
    if (rnd() % 8 == 0) m = 0xfffffffffffffull - (rnd() & 3);    // significands next to a power of two
    e = kind == 1 ? 1023 - 20 + rnd() % 40 : rnd() % 2047;
    uint64_t b = sg | e << 52 | m;
    double x;
    memcpy(&x, &b, 8);
    return x;
}
static bool same(double x, double y) { return memcmp(&x, &y, 8) == 0 || (x != x && y != y); }
extern "C" long bad_div(long n, uint64_t seed, int kind) {
    s = seed;
    long bad = 0;
    for (long i = 0; i < n; ++i) {
        const double a = val(kind), b = val(rnd() % 8 ? kind : 0);
        bad += !same(pdac_fp::div_by(a, pdac_fp::recip(b)), a / b);
    }
    return bad;
}
// quotients next to a rounding boundary: a = RN(b (q + half an ulp)) and its neighbours
extern "C" long bad_halfway(long n, uint64_t seed) {
    s = seed;
    long bad = 0;
    for (long i = 0; i < n; ++i) {
        const double b = val(1), q = val(1);
        const double h = ldexp(1.0, ilogb(q) - 53);
        double a = fma(b, q, b * h);
        for (int k = -2; k <= 2; ++k) {
            double x = a;
            for (int t = 0; t < (k < 0 ? -k : k); ++t) x = nextafter(x, k < 0 ? -INFINITY : INFINITY);
            bad += !same(pdac_fp::div_by(x, pdac_fp::recip(b)), x / b);
        }
    }
    return bad;
}
extern "C" long bad_rel(long n, uint64_t seed, int kind) {
    s = seed;
    long bad = 0;
    for (long i = 0; i < n; ++i) {
        const double a = val(kind);
        double b = val(kind);
        if (rnd() % 4) b = a + a * 1e-8 * (rnd() % 2 ? 1.0 : -1.0);       // next to the tolerance
        for (int t = rnd() % 4; t > 0; --t) b = nextafter(b, rnd() % 2 ? INFINITY : -INFINITY);
        bad += pdac_fp::rel_change_within(a, b, 1e-8) != (fabs((a - b) / a) <= 1e-8);
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("div_by")
    src = d / "t.cpp"
    src.write_text(SRC)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pdac_b200", "csrc")
    so = d / "t.so"
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-shared",
                    "-fPIC", "-I", inc, str(src), "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    for name, args in (("bad_div", [C.c_long, C.c_uint64, C.c_int]), ("bad_halfway", [C.c_long, C.c_uint64]),
                       ("bad_rel", [C.c_long, C.c_uint64, C.c_int])):
        getattr(L, name).argtypes = args
        getattr(L, name).restype = C.c_long
    return L


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_quotient_has_the_bits_of_the_division(lib, kind):
    assert lib.bad_div(400_000, 88172645463325252 + kind, kind) == 0


def test_quotients_next_to_a_rounding_boundary(lib):
    assert lib.bad_halfway(200_000, 123456789) == 0


@pytest.mark.parametrize("kind", [0, 1, 2])
def test_relative_change_decides_as_the_division(lib, kind):
    assert lib.bad_rel(400_000, 362436069 + kind, kind) == 0


REF = r"""
#include <cstdint>
#include <cstring>
#include "fpmath.h"
// pow as written with divisions, frexp and ldexp
static double exp_ref(double zh, double zl) {
    if (zh != zh) return zh;
    if (zh > 709.782712893384) return INFINITY;
    if (zh < -745.2) return 0.0;
    const double N = std::nearbyint(zh * PDAC_INV_LN2_32);
    const int n = (int)N, j = n & 31, m = (n - j) / 32;
    double r = std::fma(-N, PDAC_LN2_32_HI, zh);
    r = std::fma(-N, PDAC_LN2_32_LO, r) + zl;
    const double q = r * r * (0x1.0p-1 + r * (0x1.5555555555555p-3 + r * (0x1.5555555555555p-5 +
                     r * (0x1.1111111111111p-7 + r * 0x1.6c16c16c16c17p-10))));
    const double p = r + q, th = pdac_fp::hExp2Tab[2 * j], tl = pdac_fp::hExp2Tab[2 * j + 1], s = th + tl;
    return std::ldexp(th + (tl + s * p), m);
}
static void log_ref(double x, double &hi, double &lo) {
    int e;
    double y = std::frexp(x, &e);
    y = y * 2.0;
    e = e - 1;
    int j = (int)std::nearbyint((y - 1.0) * 128.0);
    j = j < 0 ? 0 : (j > 128 ? 128 : j);
    const double F = 1.0 + (double)j * 0x1.0p-7, f = y - F, g = f / F, gl = std::fma(-g, F, f) / F;
    const double poly = g * g * (-0x1.0p-1 + g * (0x1.5555555555555p-2 + g * (-0x1.0p-2 + g * (0x1.999999999999ap-3 +
                        g * -0x1.5555555555555p-3))));
    const double a = (double)e * PDAC_LN2_HI, b = pdac_fp::hLogTab[2 * j];
    double s1 = a + b, bb = s1 - a, t1 = (a - (s1 - bb)) + (b - bb);
    double s2 = s1 + g;
    bb = s2 - s1;
    double t2 = (s1 - (s2 - bb)) + (g - bb);
    double l = t1 + t2 + ((double)e * PDAC_LN2_LO + pdac_fp::hLogTab[2 * j + 1] + gl + poly);
    hi = s2 + l;
    lo = l - (hi - s2);
}
static double pow_ref(double x, double y) {
    if (y == 0.0 || x == 1.0) return 1.0;
    if (x != x || y != y) return x + y;
    if (x < 0.0) return NAN;  // the exponents below are no integers
    if (x == 0.0) return y > 0.0 ? 0.0 : INFINITY;
    if (x == INFINITY) return y > 0.0 ? x : 0.0;
    double lh, ll;
    log_ref(x, lh, ll);
    const double zh = y * lh, zl = std::fma(y, lh, -zh) + y * ll;
    return exp_ref(zh, zl);
}
static uint64_t s;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double any() {
    static const double special[] = {0.0, -0.0, 1.0, -2.0, INFINITY, -INFINITY, NAN, 5e-324, 2.2e-308, 1.7e308, 0.8, 10.0};
    if (rnd() % 50 == 0) return special[rnd() % 12];
    uint64_t e = rnd() % 3 ? 1023 - 30 + rnd() % 60 : rnd() % 2047, b = e << 52 | (rnd() & 0xfffffffffffffull);
    double x;
    memcpy(&x, &b, 8);
    return x;
}
static bool same(double x, double y) { return memcmp(&x, &y, 8) == 0 || (x != x && y != y); }
extern "C" long bad_pow(long n, uint64_t seed) {
    static const double ys[] = {-0.14874, 0.687f, -2.65f, 1.0 / 3.0, 0.2, 0.7, -0.25, 4.14f, 1.28f, 217.3, -309.7, 1e-3};
    s = seed;
    long bad = 0;
    for (long i = 0; i < n; ++i) {
        const double x = any();
        const pdac_fp::PowOf b = pdac_fp::pow_of(x);
        for (double y : ys) {
            const double want = pow_ref(x, y);
            bad += !same(pdac_fp::pow(x, y), want) + !same(pdac_fp::pow(b, y), want);
        }
        const double z = (double)(int64_t)rnd() * 0x1p-63 * (rnd() % 2 ? 400.0 : 3.0);
        bad += !same(pdac_fp::pow10(z), pow_ref(10.0, z)) + !same(pdac_fp::exp(z), exp_ref(z, 0.0));
        bad += !same(pdac_fp::pow10(x), pow_ref(10.0, x));
    }
    double lh, ll;
    log_ref(10.0, lh, ll);
    return bad + !same(lh, PDAC_LOGDD_10_HI) + !same(ll, PDAC_LOGDD_10_LO);
}
"""


def test_pow_has_the_bits_of_the_form_with_divisions(tmp_path):
    src = tmp_path / "p.cpp"
    src.write_text(REF)
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pdac_b200", "csrc")
    so = tmp_path / "p.so"
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-shared",
                    "-fPIC", "-I", inc, str(src), "-o", str(so)], check=True)
    L = C.CDLL(str(so))
    L.bad_pow.argtypes = [C.c_long, C.c_uint64]
    L.bad_pow.restype = C.c_long
    assert L.bad_pow(200_000, 521288629) == 0
