"""Writes the piecewise polynomials of the limiter's switch h(r).

The adiabatic limiter blends two limiters with (physics/adiabatic.hpp:692-702)

    h(r) = 1 - tanh(4 r^2 (1 - r)^0.1)   for 0 < r < 1,
    h(r) = tanh(10 (r - 1)^3)^6          for r >= 1.

h depends on r alone, so the FP64 kernels evaluate it as one polynomial of
degree 7 about the centre of the interval that r falls in (one subtraction
and seven fused multiply-adds) instead of a logarithm, two exponentials and a
division.  The intervals follow the bits of the argument, so that a shift of
its high word is the row and its centre:

    0 < r < 1    u = 1 - r, 32 intervals per power of two, 2^-40 <= u <= 1
                 (rows 0 .. 1279; h is smooth in log u, its slope unbounded at 0)
    1 <= r < 2   u = r, 256 intervals (rows 1280 .. 1535)
    2 <= r < 2.25  32 intervals (rows 1536 .. 1567); from 2.25 on h is 1 to the
                 last bit

A second table holds dh/dr in the same form, for the derivative kernels, and
a third the coefficients of h for pairs of floats (limiter_pair.cuh): the
first four as a float and its remainder, the others, whose terms are below
2^-24 of h, rounded to a float; below 1 they are those of u scaled to [1, 2).
Each polynomial interpolates at the 8 Chebyshev nodes of its interval and is
evaluated here in 45-digit decimal arithmetic; only the coefficients are
rounded.  Against the formulas at u, h is within 2.2e-16 (absolute)
and dh/dr within 5e-16 of the larger of 1 and its interval's largest value; at
r, with the rounding of 1 - r below 1/2, h is within 2.5e-16 (the formula in
doubles within 2.8e-16).
"""
from __future__ import annotations

import math
import struct
import sys
from decimal import Decimal as D, getcontext
from pathlib import Path

DEGREE = 7
OCTAVES, PER_OCTAVE = 40, 32
ROWS_BELOW = OCTAVES * PER_OCTAVE
ROWS_1_2, ROWS_2_UP = 256, 32
ROWS = ROWS_BELOW + ROWS_1_2 + ROWS_2_UP

getcontext().prec = 45


def h_below(u: D) -> tuple[D, D]:
    """(h, dh/dr) for r = 1 - u, 0 < u <= 1."""
    r = 1 - u
    p = (D("0.1") * u.ln()).exp()
    z = 8 * r * r * p
    e = z.exp()
    h = 2 / (1 + e)
    dz = 16 * r * p - D("0.8") * r * r * p / u
    return h, -h * (1 - h / 2) * dz


def h_above(r: D) -> tuple[D, D]:
    x = r - 1
    e = (20 * x * x * x).exp()
    t = (e - 1) / (e + 1)
    return t**6, 6 * t**5 * (1 - t * t) * 30 * x * x


def rows():
    """(centre, half width, formula) of every interval, in row order."""
    for k in range(OCTAVES):
        low = D(2) ** (k - OCTAVES)
        for i in range(PER_OCTAVE):
            yield low * (1 + (D(2 * i + 1) / (2 * PER_OCTAVE))), low / (2 * PER_OCTAVE), h_below
    for i in range(ROWS_1_2):
        yield 1 + D(2 * i + 1) / (2 * ROWS_1_2), D(1) / (2 * ROWS_1_2), h_above
    for i in range(ROWS_2_UP):
        yield 2 + D(2 * i + 1) / ROWS_1_2, D(1) / ROWS_1_2, h_above


def interpolate(nodes: list[D], values: list[D]) -> list[D]:
    """Monomial coefficients of the interpolating polynomial (Newton form expanded)."""
    n = len(nodes)
    c = list(values)
    for j in range(1, n):
        for i in range(n - 1, j - 1, -1):
            c[i] = (c[i] - c[i - 1]) / (nodes[i] - nodes[i - j])
    poly = [D(0)] * n
    for i in range(n - 1, -1, -1):  # poly = poly * (x - nodes[i]) + c[i]
        for k in range(n - 1, 0, -1):
            poly[k] = poly[k - 1] - nodes[i] * poly[k]
        poly[0] = c[i] - nodes[i] * poly[0]
    return poly


def tables() -> tuple[list[list[float]], list[list[float]]]:
    cheb = [D(math.cos(math.pi * (2 * j + 1) / (2 * (DEGREE + 1)))) for j in range(DEGREE + 1)]
    value, slope = [], []
    for centre, half, formula in rows():
        nodes = [half * c for c in cheb]
        got = [formula(centre + x) for x in nodes]
        value.append([float(c) for c in interpolate(nodes, [g[0] for g in got])])
        slope.append([float(c) for c in interpolate(nodes, [g[1] for g in got])])
    return value, slope


def to_float(x: float) -> float:
    return struct.unpack("f", struct.pack("f", x))[0]


def pair_row(row: list[float]) -> list[float]:
    """c0 .. c3 as a float and its remainder, then c4 .. c7 (48 bytes)."""
    out = []
    for c in row[:4]:
        out += [to_float(c), to_float(c - to_float(c))]
    return out + [to_float(c) for c in row[4:]]


def write(path: Path) -> None:
    value, slope = tables()
    lines = ["// written by limiter_table.py: rows of " + str(DEGREE + 1) + " coefficients, constant term first"]
    for name, table in (("kSwitchTable", value), ("kSwitchSlope", slope)):
        lines.append(f"SPLASH_TABLE const double {name}[{ROWS}][{DEGREE + 1}] = {{")
        lines += ["  {" + ", ".join(c.hex() for c in row) + "}," for row in table]
        lines.append("};")
    lines.append(f"SPLASH_TABLE const float kSwitchPairs[{ROWS}][12] = {{")
    for i, row in enumerate(value):
        scale = 2.0 ** (i // PER_OCTAVE - OCTAVES) if i < ROWS_BELOW else 1.0
        lines.append("  {" + ", ".join(c.hex() + "f" for c in pair_row([c * scale**k for k, c in enumerate(row)])) + "},")
    lines.append("};")
    path.write_text("\n".join(lines) + "\n")


if __name__ == "__main__":
    write(Path(sys.argv[1]))
