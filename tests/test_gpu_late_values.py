"""Host solves whose values arrive while the sources are sorted in one block (up to 16,384): the
gather of the values by itself, with the targets sorted on the second stream behind their own copy.
More than 16,384 targets, or blocks, take this route; fewer targets run on one stream."""
import numpy as np
import pytest

import treecodes as T
from tc_helpers import dev, dev_empty, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,m", [(5000, 32769), (5000, 50001), (1, 32769), (16384, 40000), (16385, 40000)])
def test_potential_host_equals_device(n, m, precision):
    r = np.random.default_rng(81 + n + m)
    xs, ys, vs = r.random(n), r.random(n), r.standard_normal(n)
    xt, yt = 1.5 * r.random(m) - 0.25, 1.5 * r.random(m) - 0.25
    ctx = T.Context(device=0, precision=precision)
    try:
        out = dev_empty(m)
        ctx.potential_device(0.5, dev(xs), dev(ys), dev(vs), dev(xt), dev(yt), out)
        for k in range(2):   # other values, same places: none of the first call's are left
            got = ctx.potential_host(0.5, xs, ys, (k + 1) * vs, xt, yt)
            assert np.array_equal(got, (k + 1) * host(out))
    finally:
        ctx.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 4096, 4097, 16384, 16385])
def test_force_host_equals_device(n, precision):
    r = np.random.default_rng(91 + n)
    xs, ys, vs = r.random(n), r.random(n), r.standard_normal(n)
    g = np.arange(4) / 4.0
    x0, y0 = np.tile(g, 4), np.repeat(g, 4)
    hs = np.full(16, 1 / 128)
    ctx = T.Context(device=0, precision=precision)
    try:
        xo, yo = dev_empty(16384), dev_empty(16384)
        ctx.force_mrag_device(0.5, dev(xs), dev(ys), dev(vs), dev(x0), dev(y0), dev(hs), xo, yo)
        for k in range(2):
            gx, gy = ctx.force_mrag_host(0.5, xs, ys, (k + 1) * vs, x0, y0, hs)
            assert np.array_equal(gx, (k + 1) * host(xo)) and np.array_equal(gy, (k + 1) * host(yo))
    finally:
        ctx.close()
