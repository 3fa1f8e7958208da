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
