"""Writes fpmath_tables.h: the table values of the exp and log routines of
fpmath.h, each the double-double (hi + lo) of the exact value, computed with
Python's decimal module at 60 significant digits.

    python pdac_b200/csrc/gen_fpmath_tables.py > pdac_b200/csrc/fpmath_tables.h
"""
import math
from decimal import Decimal, getcontext

getcontext().prec = 60


def split(v):
    hi = float(v)
    return hi, float(v - Decimal(hi))


def trimmed(v, bits):
    """v rounded down to `bits` significant bits (so that small integer
    multiples of it are exact), and the rest."""
    m, e = math.frexp(float(v))
    hi = math.ldexp(math.floor(m * 2 ** bits) / 2 ** bits, e)
    return hi, float(v - Decimal(hi))


def lit(x):
    return float.hex(x) if x != 0.0 else "0x0.0p+0"


def main():
    ln2 = Decimal(2).ln()
    out = ["// fpmath_tables.h -- generated by gen_fpmath_tables.py; do not edit.",
           "#pragma once", ""]
    hi, lo = trimmed(ln2, 42)
    out += [f"#define PDAC_LN2_HI {lit(hi)}", f"#define PDAC_LN2_LO {lit(lo)}"]
    hi, lo = trimmed(ln2 / 32, 42)
    out += [f"#define PDAC_LN2_32_HI {lit(hi)}", f"#define PDAC_LN2_32_LO {lit(lo)}",
            f"#define PDAC_INV_LN2_32 {lit(float(Decimal(32) / ln2))}", ""]
    rows = [split(Decimal(2) ** (Decimal(j) / 32)) for j in range(32)]
    out.append("// 2^(j/32), j = 0 .. 31: hi, lo")
    out.append("#define PDAC_EXP2_TABLE { \\")
    out += [f"    {lit(h)}, {lit(l)}, \\" for h, l in rows]
    out += ["}", ""]
    rows = [split((Decimal(1) + Decimal(j) / 128).ln()) for j in range(129)]
    out.append("// log(1 + j/128), j = 0 .. 128: hi, lo")
    out.append("#define PDAC_LOG_TABLE { \\")
    out += [f"    {lit(h)}, {lit(l)}, \\" for h, l in rows]
    out += ["}", ""]
    out.append("// 1 / (1 + j/128), j = 0 .. 128, rounded to nearest")
    out.append("#define PDAC_LOG_INVF_TABLE { \\")
    out += [f"    {lit(128.0 / (128.0 + j))}, \\" for j in range(129)]
    out += ["}", ""]
    print("\n".join(out))


if __name__ == "__main__":
    main()
