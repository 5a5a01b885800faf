"""Generate fixed_tables.inc, the 64-bit fixed-point tables of
fixed_geodesic.cuh: 2^(j/128) and 2^(-j/128) for j = -64..191 as integers
times 2^-61 and 2^-62, and cos and sin of 2 pi n/1024 for n = 0..1023 times
2^-62, every entry rounded to nearest.

    python raptor_gb300/csrc/gen_fixed_tables.py

Values are computed with Python's decimal module at 50 significant digits
(gen_math_tables.py), then rounded."""
import os
from decimal import Decimal

from gen_math_tables import LN2, dexp, sincospi_entry

JMIN, JMAX = -64, 192


def fixed(x, bits):
    return int((x * (1 << bits)).to_integral_value())


def main():
    here = os.path.dirname(os.path.abspath(__file__))
    out = ["// Generated by gen_fixed_tables.py - do not edit.", "",
           "// 2^(j/128) * 2^61 and 2^(-j/128) * 2^62, j = -64..191",
           f"FX_TABLE(kFxExp2, {JMAX - JMIN}) = {{"]
    for j in range(JMIN, JMAX):
        x = LN2 * Decimal(j) / 128
        out.append(f"    {{{fixed(dexp(x), 61)}ll, {fixed(dexp(-x), 62)}ll}},")
    out += ["};", "", "// sin and cos of 2 pi n / 1024, times 2^62, n = 0..1023", "FX_TABLE(kFxSinCos, 1024) = {"]
    for n in range(1024):
        s, c = sincospi_entry(n, 512)
        out.append(f"    {{{fixed(s, 62)}ll, {fixed(c, 62)}ll}},")
    out += ["};", ""]
    with open(os.path.join(here, "fixed_tables.inc"), "w") as f:
        f.write("\n".join(out))


if __name__ == "__main__":
    main()
