"""Writes fx_tables.cuh: the integer tables and constants of fx64.cuh (exp
and log on the integer pipes), each the integer nearest to the scaled exact
value (mpmath at 200 bits).  Run from this directory:
    python gen_fx_tables.py > fx_tables.cuh
"""
import mpmath

mpmath.mp.prec = 200


def q(v, bits):
    return int(mpmath.nint(v * mpmath.mpf(2) ** bits))


def main():
    ln2 = mpmath.log(2)
    step = q(ln2 / 256, 70)
    lo = (step + 2 ** 31) % 2 ** 32 - 2 ** 31
    out = ["// Generated by gen_fx_tables.py: integers nearest to the scaled exact values.",
           "#pragma once", "", "namespace dccm {", "namespace fx {", "",
           f"constexpr int EXP_INV = {q(256 / ln2, 22)};  // 256 / ln 2, 2^-22 units",
           f"constexpr int EXP_STEP_H = {(step - lo) >> 32};  // ln 2 / 256 in 2^-70 units, high word",
           f"constexpr int EXP_STEP_L = {lo};  // and signed low word",
           f"constexpr unsigned long long LN2_57 = {q(ln2, 57)}ull;  // ln 2, 2^-57 units", "",
           "// 2^(j / 256), j = 0 .. 255, 2^-62 units",
           "__device__ const unsigned long long EXP2_256[256] = {"]
    out += [f"    {q(mpmath.power(2, mpmath.mpf(j) / 256), 62)}ull," for j in range(256)]
    out += ["};", "",
            "// {1 / F in 2^-63 units, ln F in 2^-57 units} for F = 1 + j / 256, j = 0 .. 255",
            "__device__ const ulonglong2 LOG_256[256] = {"]
    for j in range(256):
        F = 1 + mpmath.mpf(j) / 256
        out.append(f"    {{{q(1 / F, 63)}ull, {q(mpmath.log(F), 57)}ull}},")
    out += ["};", "", "}  // namespace fx", "}  // namespace dccm", ""]
    print("\n".join(out))


if __name__ == "__main__":
    main()
