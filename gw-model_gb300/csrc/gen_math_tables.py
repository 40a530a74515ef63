"""Generates gw_math_tables.h: the constants of the engine's FP64 exp and log (gw_math64.cuh), which
run in 64-bit integer arithmetic.

exp: 2^(j/256), j = 0..255, as integers of 63 fractional bits, 1/ln2 and the Taylor coefficients
ln2^k / k! of 2^t.
log: for j = 0..255, c_j = 2^16 / (1 + j/256) rounded up to an integer, and -log(c_j / 2^16) with 64
fractional bits; ln2; the magnitudes 1 / k of the coefficients of log(1 + u).
All values come from 80-digit decimal arithmetic (Python's decimal module).

Usage: python gen_math_tables.py > gw_math_tables.h
"""
from decimal import ROUND_CEILING, ROUND_HALF_EVEN, Decimal, getcontext

getcontext().prec = 80


def fixed(d: Decimal, bits: int) -> int:
    return int((d * Decimal(2) ** bits).to_integral_value(rounding=ROUND_HALF_EVEN))


def main():
    ln2 = Decimal(2).ln()
    out = ["// gw_math_tables.h -- generated by gen_math_tables.py; do not edit.", "#pragma once", "namespace gw {",
           "namespace math64 {"]
    out.append(f"constexpr unsigned long long kLog2e63 = {fixed(1 / ln2, 63):#x}ull;  // 1/ln2, 63 fractional bits")
    out.append(f"constexpr unsigned long long kLn2 = {fixed(ln2, 64):#x}ull;      // ln2, 64 fractional bits")
    bias = 2048 * fixed(ln2, 64)
    out.append("// 2048 times that, as two words")
    out.append(f"constexpr unsigned long long kLn2BiasHi = {bias >> 64:#x}ull, kLn2BiasLo = {bias & (2**64 - 1):#x}ull;")
    f = Decimal(1)
    for k in range(1, 6):
        f *= ln2 / k
        if k <= 3:
            out.append(f"constexpr unsigned long long kExp{k} = {fixed(f, 64):#x}ull;  // ln2^{k}/{k}!, 64 fractional bits")
        else:
            out.append(f"constexpr unsigned int kExp{k} = {fixed(f, 32):#x}u;  // ln2^{k}/{k}!, 32 fractional bits")
    for k in range(2, 8):
        if k <= 3:
            out.append(f"constexpr unsigned long long kLog{k} = {fixed(Decimal(1) / k, 64):#x}ull;  // 1/{k}, 64 fractional bits")
        else:
            out.append(f"constexpr unsigned int kLog{k} = {fixed(Decimal(1) / k, 32):#x}u;  // 1/{k}, 32 fractional bits")
    out += ["// 2^(j/256), 63 fractional bits", "#define GW_EXP2_TABLE \\", "    { \\"]
    for j in range(0, 256, 4):
        out.append("        " + " ".join(f"{fixed((Decimal(j + i) / 256 * ln2).exp(), 63):#x}ull," for i in range(4)) + " \\")
    out += ["    }", "// {c_j, -log(c_j / 2^16) with 64 fractional bits}", "#define GW_LOG_TABLE \\", "    { \\"]
    for j in range(0, 256, 2):
        row = []
        for i in range(2):
            c = int((65536 / (1 + Decimal(j + i) / 256)).to_integral_value(rounding=ROUND_CEILING))
            row.append(f"{{{c}ull, {fixed(-(Decimal(c) / 65536).ln(), 64):#x}ull}},")
        out.append("        " + " ".join(row) + " \\")
    out += ["    }", "}  // namespace math64", "}  // namespace gw"]
    print("\n".join(out))


if __name__ == "__main__":
    main()
