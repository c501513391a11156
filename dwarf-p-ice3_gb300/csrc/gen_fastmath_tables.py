"""Generate fastmath_tables.h: the tables and split constants of the FP64
exp/exp10/log in fastmath.cuh, computed in 200-bit arithmetic with mpmath
and rounded to nearest.

    python dwarf-p-ice3_gb300/csrc/gen_fastmath_tables.py

exp (after Tang, ACM TOMS 15(2), 1989, in fixed point): 2^(j/512), j = 0..511,
as a 64-bit integer times 2^-62; ln2/512 and log10(2)/512 as a 64-bit integer
times 2^-70 and 32 further bits, and 2^20 times each modulo 2^-6 (the bias
that keeps the multiple positive).

atan (table-driven reduction in the manner of Tang's methods): atan(j/64) and
pi/2 - atan(j/64), j = 0..64, as 64-bit integers times 2^-64 and 2^-62.

log (after Tang, ACM TOMS 16(4), 1990, in fixed point): the significand z in
[1, 2) is split into 512 intervals by its 9 leading fraction bits; per
interval [z0, z0 + 1/512) the integer c = ceil(2048/z0), so that r = z c/2048
- 1 is exact in 64 bits and not negative (r < 2^-8.4), and -log(c/2048) -
1100 ln2 as a 96-bit integer times 2^-72 (the bias keeps the exponent's
multiple of ln2 positive).
"""
from __future__ import annotations

import os

import mpmath as mp
import numpy as np

mp.mp.prec = 200
HERE = os.path.dirname(os.path.abspath(__file__))


def dbl(x) -> float:
    return float(mp.mpf(x))          # round to nearest double


def flt(x) -> float:
    return float(np.float32(dbl(x)))  # nearest float (values here are far from float ties)


def fix(x, bits: int) -> int:
    """x 2^bits rounded to an integer."""
    return int(mp.nint(mp.mpf(x) * mp.mpf(2) ** bits))


def words(n: int, count: int):
    """The 32-bit words of n modulo 2^(32 count), lowest first."""
    return [(n >> (32 * i)) & 0xffffffff for i in range(count)]


def fhex(v: float) -> str:
    return f"{v.hex()}f" if v != 0.0 else "0.0f"


def main() -> None:
    lines = ["// Generated by gen_fastmath_tables.py (mpmath, 200-bit) - do not edit.",
             "#pragma once", "",
             "// 2^(j/512) 2^62, j = 0..511",
             "#define FM_EXP_TABLE_INIT { \\"]
    for j in range(512):
        lines.append(f"  {fix(mp.mpf(2) ** (mp.mpf(j) / 512), 62):#018x}ull, \\")
    lines += ["}", "",
              "// per 9-bit significand interval: {c, (-log(c/2048) - 1100 ln2) 2^72 in three words, lowest first}",
              "#define FM_LOG_TABLE_INIT { \\"]
    for i in range(512):
        c = -(-2048 * 512 // (512 + i))
        w = words(fix(-mp.log(mp.mpf(c) / 2048) - 1100 * mp.log(2), 72), 3)
        lines.append(f"  {{{c}u, {w[0]:#010x}u, {w[1]:#010x}u, {w[2]:#010x}u}}, \\")
    lines += ["}", "",
              "// {atan(j/64) 2^64, (pi/2 - atan(j/64)) 2^62}, j = 0..64",
              "#define FM_ATAN_TABLE_INIT { \\"]
    for j in range(65):
        t = mp.atan(mp.mpf(j) / 64)
        lines.append(f"  {{{fix(t, 64):#018x}ull, {fix(mp.pi / 2 - t, 62):#018x}ull}}, \\")
    lines += ["}", ""]
    l512 = mp.log(2) / 512
    lg512 = mp.log10(2) / 512
    ln2 = words(fix(mp.log(2), 72), 3)
    consts = {
        "FM_INV_L512_F": fhex(flt(512 / mp.log(2))), "FM_INV_LG512_F": fhex(flt(512 / mp.log10(2))),
        "FM_LN10_62": f"{fix(mp.log(10), 62):#018x}ull",
        "FM_LN2_W0": f"{ln2[0]:#010x}u", "FM_LN2_W1": f"{ln2[1]:#010x}u", "FM_LN2_W2": f"{ln2[2]}u",
        "FM_PIO2": dbl(mp.pi / 2).hex(),
    }
    for name, v in (("L512", l512), ("LG512", lg512)):
        f102 = fix(v, 102)
        consts[f"FM_{name}_HI"] = f"{f102 >> 32:#018x}ull"               # 2^-70 units
        consts[f"FM_{name}_LO"] = f"{f102 & 0xffffffff:#010x}u"          # the next 32 bits
        consts[f"FM_{name}_BIAS"] = f"{fix(v * 2 ** 20, 70) % 2 ** 64:#018x}ull"
    for k, v in consts.items():
        lines.append(f"#define {k} {v}")
    with open(os.path.join(HERE, "fastmath_tables.h"), "w") as f:
        f.write("\n".join(lines) + "\n")


if __name__ == "__main__":
    main()
