"""Expansions across distances whose squares near or pass the top of the number range: the
translations' reciprocals hold there too (rcp_any in tc_common.cuh)."""
import numpy as np
import pytest

import treecodes as T
from tc_helpers import dev, dev_empty, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [12, 24])
@pytest.mark.parametrize("far", [1e150, 1e153, 9e153, 1.3e154, 2e154, 1e300])
@pytest.mark.parametrize("nblocks", [1, 600])   # a block per brick, and (9600 bricks) a warp
def test_local_expansion_of_distant_cells(nblocks, far, order):
    """One block near the sources, the others far from them: one E2L each, the field m / d."""
    r = np.random.default_rng(31)
    n = 300
    xs, ys, vs = r.random(n), r.random(n), r.random(n)
    x0 = np.full(nblocks, far)
    y0 = np.zeros(nblocks)
    hs = np.full(nblocks, 0.01)
    xo, yo = dev_empty(1024 * nblocks), dev_empty(1024 * nblocks)
    ctx = T.Context(device=0)
    try:
        ctx.set_orders(force_order=order)
        ctx.force_mrag_device(0.5, dev(xs), dev(ys), dev(vs), dev(x0), dev(y0), dev(hs), xo, yo)
        assert ctx.stats()["n_e2l"] == 16 * nblocks
    finally:
        ctx.close()
    xo, yo = host(xo), host(yo)
    # an overflowing square leaves no field; otherwise m / d = m d / d^2, to the roundings of the sum
    # and the expansion, and to 2^-1075 in a reciprocal of d^2 below 2^-1022
    want = vs.sum() / far if far < 1.34e154 else 0.0
    bound = (n + 20) * 2.0 ** -52 * want + (vs.sum() * far * 2.0 ** -1073 if want else 0.0)
    assert np.all(np.abs(xo - want) <= bound)
    assert np.all(np.abs(yo) <= 1e-140)


def test_merged_expansion_of_distant_cells():
    """Two opposite clusters 2 h = 2^505 apart: their common cell has no mass, so its potential at
    distance d = 31 h is the dipole's, log((d + h) / (d - h)) = 2 h / d (1 + (h / d)^2 / 3 + ..)."""
    n, a, z = 1024, 2.0 ** 505, 2.0 ** 509
    xs = np.r_[np.zeros(n), np.full(n, a)]
    vs = np.r_[np.ones(n), -np.ones(n)]
    out = dev_empty(1)
    ctx = T.Context(device=0)
    try:
        ctx.potential_device(0.5, dev(xs), dev(0 * xs), dev(vs), dev([z]), dev([0.0]), out)
        assert ctx.stats()["n_e2p"] == 1
    finally:
        ctx.close()
    want = -n * np.log1p(-a / z)
    h = 0.5 * a
    # (the second and higher coefficients are outside the number range and left out)
    assert abs(host(out)[0] - want) <= 2 * (h / (z - h)) ** 2 / 3 * want
