"""Writes pow_fx_tables.inc, the fixed-point tables of pow_exner_fx.cuh, from exact decimal
arithmetic.

* log table, j = 0..1023: n_j / 2^11, the multiple of 2^-11 nearest to 1 / c_j with c_j = 1 +
  (j + 1/2) / 1024 (1025 / 2^11 for the last, whose nearest is 1/2), and -log2(n_j / 2^11) as 96
  fraction bits;
* exp table, j = 0..1023: 2**(j / 1024) as 95 fraction bits;
* 1 / ln 2 on 63 and ln 2 on 64 fraction bits, 1 / (n ln 2) (n = 2..7) and 1 / n! (n = 3..6).

Every entry is the nearest integer of a 60-digit decimal (Python's decimal module rounds ln and
power correctly at its context precision).

Run:  python mpas_dycore_pytorch_gb300/csrc/gen_pow_fx_tables.py  (rewrites pow_fx_tables.inc)
"""

from __future__ import annotations

import pathlib
import sys
from decimal import ROUND_HALF_EVEN, Decimal, getcontext

getcontext().prec = 60
HERE = pathlib.Path(__file__).resolve().parent
LN2 = Decimal(2).ln()


def fixed(d: Decimal, bits: int) -> int:
    return int((d * 2 ** bits).to_integral_value(ROUND_HALF_EVEN))


def render() -> str:
    lines = ["// Generated by gen_pow_fx_tables.py from 60-digit decimal arithmetic; do not edit.",
             "// {n, -log2(n / 2^11): 32 and 64 fraction bits}", "MPASG_POWFX_TABLE Entry kPowFxLog[1024] = {"]
    row = []
    for j in range(1024):
        c = Decimal(1) + (Decimal(j) + Decimal("0.5")) / 1024
        n = max(1025, fixed(1 / c, 11))
        t = fixed(-(Decimal(n) / 2 ** 11).ln() / LN2, 96)
        row.append(f"{{0x{t & (2 ** 64 - 1):x}u, {n}u, 0x{t >> 64:x}u}}")
    lines += ["  " + ", ".join(row[i:i + 3]) + "," for i in range(0, 1024, 3)]
    lines += ["};", "// {2^(j/1024): 63 fraction bits, the next 32}", "MPASG_POWFX_TABLE Entry kPowFxExp[1024] = {"]
    row = []
    for j in range(1024):
        t = fixed(Decimal(2) ** (Decimal(j) / 1024), 95)
        row.append(f"{{0x{t >> 32:x}u, 0x{t & (2 ** 32 - 1):x}u, 0u}}")
    lines += ["  " + ", ".join(row[i:i + 3]) + "," for i in range(0, 1024, 3)]
    lines.append("};")
    lines.append(f"constexpr uint64_t kPowFxInvLn2 = 0x{fixed(1 / LN2, 63):x}u;")
    lines.append(f"constexpr uint64_t kPowFxLn2 = 0x{fixed(LN2, 64):x}u;")
    for n, bits in ((2, 64), (3, 64), (4, 64), (5, 32), (6, 32), (7, 32)):
        lines.append(f"constexpr uint{bits}_t kPowFxC{n} = 0x{fixed(1 / (n * LN2), bits):x}u;")
    for n, f, bits in ((3, 6, 64), (4, 24, 64), (5, 120, 32), (6, 720, 32)):
        lines.append(f"constexpr uint{bits}_t kPowFxD{n} = 0x{fixed(Decimal(1) / f, bits):x}u;")
    return "\n".join(lines) + "\n"


if __name__ == "__main__":
    text = render()
    if len(sys.argv) > 1 and sys.argv[1] == "--check":
        sys.exit(0 if (HERE / "pow_fx_tables.inc").read_text() == text else 1)
    (HERE / "pow_fx_tables.inc").write_text(text)
