#!/usr/bin/env python
"""Regenerates tc_near_log_table.cuh: the table and the polynomial of log_near (tc_math.cuh).

log_near splits x = 2^e m, m in [0.7066, 1.4133), takes the NBITS = 9 fraction bits of m below
its offset high word as a table index, and

    log x = e ln 2 + (-log c) + log1p(r),   r = m c - 1,   log1p(r) = r (1 + r q(r)).

Entry i holds (c, -log c): c is the double nearest to the reciprocal of the middle of the m that
share the index, and -log c is rounded to double.  The offset BASE puts m = 1 inside an interval,
(1 - 2^-11, 1 + 2^-10), whose c is exactly 1, so that the result keeps its relative precision near
x = 1.  |r| <= 2^-10 everywhere; r is one fma, so its rounding is relative to r itself.  q is the
degree-3 interpolant of (log1p(r) - r) / r^2 at the 4 first-kind Chebyshev nodes of
[-2^-10, 2^-10].  Everything is computed with 50 significant digits (mpmath) and rounded to the
nearest double.

Run it to rewrite tc_near_log_table.cuh beside this file (`--check` compares instead).
"""
import os
import struct
import sys

import mpmath as mp

NBITS = 9
NTAB = 1 << NBITS
BASE = 0x3fe69c00                        # high word of the smallest m
STEP = 1 << (20 - NBITS)                 # high-word units per entry
DEGREE = 3
R_MAX = mp.mpf(2) ** -10
HEADER = os.path.join(os.path.dirname(os.path.abspath(__file__)), "tc_near_log_table.cuh")


def m_at(high):
    """The double whose high word is `high` (0x3fe..... or 0x3ff.....) and low word 0."""
    return mp.mpf(struct.unpack("<d", struct.pack("<Q", high << 32))[0])


def table(digits=50):
    """(c, -log c) of every entry."""
    out = []
    with mp.workdps(digits):
        for i in range(NTAB):
            lo, hi = m_at(BASE + i * STEP), m_at(BASE + (i + 1) * STEP)
            c = 1.0 if lo < 1 < hi else float(2 / (lo + hi))
            out.append((c, float(-mp.log(mp.mpf(c))) if c != 1.0 else 0.0))
    return out


def q_exact(r):
    """(log1p(r) - r) / r^2; its series -1/2 + r/3 - r^2/4 + ... next to 0."""
    if abs(r) < mp.mpf(2) ** -40:
        return sum((-1) ** (k + 1) * r ** k / (k + 2) for k in range(8))
    return (mp.log1p(r) - r) / (r * r)


def coefficients(degree=DEGREE, digits=50):
    """Coefficients q_0..q_degree (double) of the interpolant, constant term first."""
    with mp.workdps(digits):
        n = degree + 1
        nodes = [R_MAX * mp.cos((2 * k + 1) * mp.pi / (2 * n)) for k in range(n)]
        a = mp.matrix(n, n)
        b = mp.matrix(n, 1)
        for i, r in enumerate(nodes):
            for j in range(n):
                a[i, j] = r ** j
            b[i] = q_exact(r)
        c = mp.lu_solve(a, b)
        return [float(c[j]) for j in range(n)]


def header_text():
    lines = [
        "// tc_near_log_table.cuh -- written by fit_near_log_table.py (do not edit): the table and",
        "// the polynomial of log_near in tc_math.cuh.",
        "#pragma once",
        "",
        "namespace tc {",
        "",
        f"constexpr int NLOG_BASE = 0x{BASE:08x};   // high word of the smallest m",
        f"constexpr int NLOG_BITS = {NBITS};",
        f"constexpr int NLOG_NTAB = {NTAB};",
        "",
        f"// log1p(r) = r (1 + r q(r)) on |r| <= 2^-10; q_0 .. q_{DEGREE}",
    ]
    for j, c in enumerate(coefficients()):
        lines.append(f"constexpr double NLOG_Q{j} = {c.hex()};")
    lines += ["", "// (c, -log c), c the reciprocal of the middle of entry i's m",
              "static __device__ const double2 NLOG_TAB[NLOG_NTAB] = {"]
    for c, t in table():
        lines.append(f"    {{{c.hex()}, {t.hex()}}},")
    lines += ["};", "", "}  // namespace tc", ""]
    return "\n".join(lines)


if __name__ == "__main__":
    text = header_text()
    if "--check" in sys.argv:
        ok = open(HEADER).read() == text
        print("tc_near_log_table.cuh is", "current" if ok else "STALE")
        sys.exit(0 if ok else 1)
    with open(HEADER, "w") as f:
        f.write(text)
    print("wrote", HEADER)
