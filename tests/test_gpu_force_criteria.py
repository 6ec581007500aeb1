"""The force traversal's own decisions (classify in force.cu): the list sizes of a solve equal those of
a walk over the same tree that takes the reference's square root and division at every node
(drivers/treecode-force.cpp:136-151), for bricks anywhere and for bricks whose distance from a cell
is within some units in the last place of the E2L border."""
import math
from fractions import Fraction

import numpy as np
import pytest

import treecodes as T
from tc_helpers import dev, dev_empty

pytestmark = pytest.mark.gpu


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def walk(t, x0, y0, h, theta):
    """E2L, E2P and P2P list sizes of one 8 x 8 brick."""
    inv, theta2 = 1.0 / theta, theta * theta
    cx, cy = fma(3.5, h, x0), fma(3.5, h, y0)
    rbrick = 4.949747468305833 * h
    xlo, xhi, ylo, yhi = x0, fma(7.0, h, x0), y0, fma(7.0, h, y0)
    sizes, stack = [0, 0, 0], [0]
    while stack:
        i = stack.pop()
        r, xc, yc = float(t["r"][i]), float(t["xcom"][i]), float(t["ycom"][i])
        dx, dy = cx - xc, cy - yc
        dist = math.sqrt(fma(dx, dx, dy * dy))
        ratio = dist / r if r else (math.inf if dist else math.nan)
        if ratio - 1.0 > inv and rbrick <= r:
            sizes[0] += 1
            continue
        ex = max(xlo, min(xhi, xc)) - xc
        ey = max(ylo, min(yhi, yc)) - yc
        if r * r < theta2 * fma(ex, ex, ey * ey):
            sizes[1] += 1
        elif t["child"][i] < 0:
            sizes[2] += int(t["count"][i] > 0)
        else:
            stack += range(t["child"][i], t["child"][i] + 4)
    return sizes


@pytest.mark.parametrize("theta", [0.3, 0.5, 1.0])
def test_list_sizes_equal_the_exact_walk(theta):
    r = np.random.default_rng(101)
    n = 6000
    xs, ys, vs = r.random(n), r.random(n) ** 2, r.standard_normal(n)
    ctx = T.Context(device=0)
    try:
        ctx.set_blocksize(8)
        t = ctx.tree("force", dev(xs), dev(ys), dev(vs))
        x0, y0, hs = list(r.random(150)), list(r.random(150)), [1 / 256] * 150
        cells = [i for i in np.flatnonzero(t["r"] > 0) if t["r"][i] > 5e-3]
        for i in r.choice(cells, 100):   # around the border of a cell
            reach = float(t["r"][i]) * (1 + 1 / theta)
            a = r.uniform(0, 2 * np.pi)
            d = reach * (1 + float(r.choice([-1, 1]) * 10.0 ** r.uniform(-16.5, -11)))
            h = 2.0 ** -14
            x0.append(float(t["xcom"][i]) + d * np.cos(a) - 3.5 * h)
            y0.append(float(t["ycom"][i]) + d * np.sin(a) - 3.5 * h)
            hs.append(h)
        want = np.sum([walk(t, *b, theta) for b in zip(x0, y0, hs)], axis=0)
        xo, yo = dev_empty(64 * len(hs)), dev_empty(64 * len(hs))
        ctx.force_mrag_device(theta, dev(xs), dev(ys), dev(vs), dev(x0), dev(y0), dev(hs), xo, yo)
        st = ctx.stats()
    finally:
        ctx.close()
    assert [st["n_e2l"], st["n_e2p"], st["n_p2p"]] == list(want)
