"""Potentials over distances near the top of the number range.  The FP64 evaluation's logarithm
(log_near in tc_math.cuh), its bit arithmetic restated as the kernel has it, holds from 2^-1022 to
2^NLOG_TOP; solves whose squared distances may be larger, or overflow, take the logarithm that holds
for every argument, with log(infinity) = 1024 ln 2."""
import math
import os
import re
import struct
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "2d-treecodes_b200", "csrc")
SRC = open(os.path.join(CSRC, "tc_near_log_table.cuh")).read()
MATH = open(os.path.join(CSRC, "tc_math.cuh")).read()
COMMON = open(os.path.join(CSRC, "tc_common.cuh")).read()
BASE = int(re.search(r"NLOG_BASE = (0x[0-9a-f]+);", SRC).group(1), 16)
BITS = int(re.search(r"NLOG_BITS = (\d+);", SRC).group(1))
Q = [float.fromhex(h) for h in re.findall(r"NLOG_Q\d = (-?0x[0-9a-fp.+-]+);", SRC)]
TAB = [(float.fromhex(a), float.fromhex(b)) for a, b in
       re.findall(r"\{(0x[0-9a-fp.+-]+), (-?0x[0-9a-fp.+-]+)\}", SRC)]
LN2 = float.fromhex("0x1.62e42fefa39efp-1")
LOG_INF = 1024 * math.log(2.0)


def top():
    return int(re.search(r"NLOG_TOP = (\d+);", MATH).group(1))


def reach():
    return float.fromhex(re.search(r"NEAR_REACH = (0x[0-9a-fp.+-]+);", COMMON).group(1))


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def log_near(x):
    """The kernel's steps: the high word of c less x's exponent, as 32-bit integers."""
    hi = struct.unpack("<Q", struct.pack("<d", x))[0] >> 32
    ix = hi - BASE
    e = ix >> 20
    c, t0 = TAB[(ix >> (20 - BITS)) & ((1 << BITS) - 1)]
    cb = struct.unpack("<Q", struct.pack("<d", c))[0]
    chi = ((cb >> 32) - (ix & 0xfff00000)) & 0xffffffff
    c = struct.unpack("<d", struct.pack("<Q", (chi << 32) | (cb & 0xffffffff)))[0]
    r = fma(x, c, -1.0)
    t = Q[3]
    for q in (Q[2], Q[1], Q[0], 1.0):
        t = fma(t, r, q)
    return fma(float(e), LN2, fma(t, r, t0))


def test_log_near_over_its_range():
    mp = pytest.importorskip("mpmath")
    # the largest squared distance of a solve that takes log_near: both offsets below the reach
    assert 2 * Fraction(reach()) ** 2 + 1 < Fraction(2) ** top()
    r = np.random.default_rng(21)
    xs = list(2.0 ** r.uniform(-1022, top(), 1500)) + [2.0 ** -1022, 2.0 ** -52 * 10, 2.0 * reach() ** 2]
    for k in range(0, 1 << BITS, 3):   # ends of the table's intervals at both ends of the range
        m = struct.unpack("<d", struct.pack("<Q", (BASE + (k << (20 - BITS))) << 32))[0]
        for e in (-1021, 0, top() - 2):
            xs += [m * 2.0 ** e, np.nextafter(m * 2.0 ** e, 0)]
    with mp.workdps(40):
        for x in xs:
            x = float(x)
            exact = mp.log(mp.mpf(x))
            assert abs(mp.mpf(log_near(x)) - exact) < 2 * math.ulp(abs(float(exact))), x


def logs(xt, yt, xs, ys):
    """log(r^2 + 10 eps) of every pair, an overflow giving 1024 ln 2."""
    with np.errstate(over="ignore"):
        dx, dy = xt[:, None] - xs[None], yt[:, None] - ys[None]
        return np.minimum(np.log(dx * dx + dy * dy + 10 * 2.0 ** -52), LOG_INF)


FAR = np.array([2.0 ** 508, 2.0 ** 509, 2.0 ** 510, 5e153, 8e153, 1e154, 1.3e154, 2e154, 1e160, 1e200,
                1e299, 1e301, 1e307, -8e153, -1e154, -1e300])


def solve(theta, xs, ys, vs, xt, yt):
    import torch
    import treecodes as T
    dev = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")
    out = torch.empty(len(xt), device="cuda", dtype=torch.float64)
    ctx = T.Context(device=0)
    try:
        args = [dev(a) for a in (xs, ys, vs, xt, yt)]
        torch.cuda.synchronize()
        ctx.potential_device(theta, *args, out)
    finally:
        ctx.close()
    return out.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("theta", [1e-300, 0.5], ids=["near", "far"])
@pytest.mark.parametrize("n,more", [(2, 0), (200, 0), (1000, 0), (200, 40000), (20000, 100),
                                    (20000, 40000)])   # every target sort
def test_targets_at_the_top_of_the_range(theta, n, more):
    """Far from every source each cell's potential is its mass times log r; the near field (no cell
    is accepted at so small a theta) sums the same logarithms."""
    r = np.random.default_rng(22 + n)
    xs, ys, vs = r.random(n), r.random(n), r.standard_normal(n)
    xt, yt = FAR, FAR[::-1] * 0.25
    k = len(xt)
    if theta < 1e-9 and n <= 1000:   # with targets among the sources, compared too
        k += 50
        xt, yt = np.r_[xt, r.random(50)], np.r_[yt, r.random(50)]
    got = solve(theta, xs, ys, vs, np.r_[xt, r.random(more)], np.r_[yt, r.random(more)])
    assert np.all(np.isfinite(got))
    got = got[:k]
    want_terms = vs[None] * logs(xt, yt, xs, ys)
    # 2 ulp of each logarithm, n roundings of the sum
    bound = (n + 4) * 2.0 ** -52 * np.abs(want_terms).sum(1) * 0.5
    assert np.all(np.abs(got - 0.5 * want_terms.sum(1)) <= bound)


@pytest.mark.gpu
@pytest.mark.parametrize("where", [5e153, 1e154, 1e160, 1e300])
def test_common_far_field_of_a_cell_at_the_top_of_the_range(where):
    """262,144 and more targets share far fields: a lone source far beyond them is in every set's."""
    r = np.random.default_rng(23)
    xs, ys, vs = np.r_[r.random(100), where], np.r_[r.random(100), 0.5], np.r_[r.random(100), 0.75]
    m = 262144 + 77
    xt, yt = r.random(m), r.random(m)
    pick = r.integers(0, m, 2000)
    terms = 0.5 * vs[None] * logs(xt[pick], yt[pick], xs, ys)
    got = solve(0.5, xs, ys, vs, xt, yt)[pick]
    # the truncation of 12 terms at r / d < 1/2, and the roundings of the sum
    cut = np.abs(vs).sum() * 0.5 ** 13 / (13 * 0.5)
    bound = cut + len(vs) * 2.0 ** -52 * np.abs(terms).sum(1)
    assert np.all(np.abs(got - terms.sum(1)) <= bound)
