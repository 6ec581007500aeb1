"""The FP64 potential evaluation's logarithm (log_near in tc_math.cuh): its table and polynomial are
what fit_near_log_table.py writes, the algorithm restated with exact fused multiply-adds is within
2 ulp of log x, and on the GPU the P2P of a single unit source gives log(r^2 + 10 eps) / 2."""
import math
import os
import re
import struct
import sys
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "2d-treecodes_b200")
CSRC = os.path.join(PKG, "csrc")
HEADER = os.path.join(CSRC, "tc_near_log_table.cuh")
sys.path.insert(0, PKG)

SRC = open(HEADER).read()
BASE = int(re.search(r"NLOG_BASE = (0x[0-9a-f]+);", SRC).group(1), 16)
BITS = int(re.search(r"NLOG_BITS = (\d+);", SRC).group(1))
Q = [float.fromhex(h) for h in re.findall(r"NLOG_Q\d = (-?0x[0-9a-fp.+-]+);", SRC)]
TAB = [(float.fromhex(a), float.fromhex(b)) for a, b in
       re.findall(r"\{(0x[0-9a-fp.+-]+), (-?0x[0-9a-fp.+-]+)\}", SRC)]
LN2 = float.fromhex("0x1.62e42fefa39efp-1")


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def log_near(x):
    u = struct.unpack("<Q", struct.pack("<d", x))[0]
    hi, lo = u >> 32, u & 0xffffffff
    ix = hi - BASE
    e = ix >> 20
    m = struct.unpack("<d", struct.pack("<Q", ((hi - (e << 20)) << 32) | lo))[0]
    c, t0 = TAB[(ix >> (20 - BITS)) & ((1 << BITS) - 1)]
    r = fma(m, c, -1.0)
    t = Q[-1]
    for q in Q[-2::-1] + [1.0]:
        t = fma(t, r, q)
    return fma(float(e), LN2, fma(t, r, t0)), r


def arguments():
    r = np.random.default_rng(12)
    xs = list(np.exp(r.uniform(np.log(2e-15), np.log(1e6), 1500)))
    for b in [1.0, 2.0, 0.5, 2.0 ** -40, 2.0 ** 19, math.sqrt(2.0), math.sqrt(0.5)]:
        xs += [b, np.nextafter(b, 0), np.nextafter(b, 4 * b)]
        xs += list(b * (1 + np.linspace(-4e-3, 4e-3, 81)))
    # both ends of every table interval, and the largest and smallest normal numbers
    for i in range((1 << BITS) + 1):
        m = struct.unpack("<d", struct.pack("<Q", (BASE + (i << (20 - BITS))) << 32))[0]
        xs += [m, np.nextafter(m, 0)]
    xs += [float.fromhex("0x1p-1022"), float.fromhex("0x1.fffffffffffffp+1023")]
    return [float(x) for x in xs]


def test_table_regenerates():
    pytest.importorskip("mpmath")
    sys.path.insert(0, CSRC)
    try:
        import fit_near_log_table
    finally:
        sys.path.remove(CSRC)
    assert SRC == fit_near_log_table.header_text()


def test_log_near_within_two_ulp_of_the_exact_log():
    mp = pytest.importorskip("mpmath")
    assert len(TAB) == 1 << BITS
    worst = rmax = 0.0
    with mp.workdps(40):
        for x in arguments():
            got, r = log_near(x)
            exact = mp.log(mp.mpf(x))
            ref = float(exact)
            ulp = math.ulp(abs(ref)) if ref != 0 else math.ulp(0.0)
            worst = max(worst, float(abs(mp.mpf(got) - exact)) / ulp)
            rmax = max(rmax, abs(r))
    assert rmax <= 2.0 ** -10, rmax
    assert worst < 2.0, worst


@pytest.mark.gpu
def test_p2p_of_one_source_is_the_log():
    import torch
    import treecodes as T

    r = np.random.default_rng(13)
    d = np.concatenate([np.exp(r.uniform(np.log(1e-9), np.log(1e3), 40000)),
                        1 + np.linspace(-4e-3, 4e-3, 4001), [0.0]])
    # a source at the origin and another of zero value give the tree an extent; theta = 1e-9 keeps
    # every target in the near field
    dev = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device="cuda")
    out = torch.empty(len(d), device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    T.Context().potential_device(1e-9, dev([0.0, 1.0]), dev([0.0, 1.0]), dev([1.0, 0.0]), dev(d),
                                 dev(0 * d), out)
    x = np.array([fma(float(v), float(v), 10 * 2.0 ** -52) for v in d])   # the kernel's argument
    ref = 0.5 * np.log(x)
    # 2 ulp of log_near and numpy's 1, with one rounding of the sum
    assert np.all(np.abs(out.cpu().numpy() - ref) <= 4 * np.spacing(np.abs(ref)))
