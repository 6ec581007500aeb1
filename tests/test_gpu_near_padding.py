"""The force's near field on tiles that 32 sources do not fill, far from the origin: the lanes past
the tile must not bring a place of their own into the sums (squares of 1e80 overflow in products)."""
import numpy as np
import pytest

import treecodes as T
from tc_helpers import dev, dev_empty, host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("base", [0.0, 2.0 ** 200, 2.0 ** 266, -2.0 ** 300])
@pytest.mark.parametrize("n", [1, 3, 31, 33, 63, 65])
def test_ragged_tiles_far_from_the_origin(n, base):
    r = np.random.default_rng(41 + n)
    unit = 2.0 ** 233 if abs(base) > 2.0 ** 250 else (2.0 ** 160 if base else 1.0)
    # places that doubles hold exactly, sources between the targets
    xs = base + (r.integers(0, 512, n) + 0.5) * unit
    ys = base + (r.integers(0, 512, n) + 0.5) * unit
    vs = r.standard_normal(n)
    h = 16 * unit
    q = np.arange(32)
    xt, yt = np.tile(base + q * h, 32), np.repeat(base + q * h, 32)
    dx, dy = xt[:, None] - xs[None], yt[:, None] - ys[None]
    f = vs / (dx * dx + dy * dy + 10 * 2.0 ** -52)
    xo, yo = dev_empty(1024), dev_empty(1024)
    ctx = T.Context(device=0)
    try:
        # (no cell is far at this theta)
        ctx.force_mrag_device(1e-6, dev(xs), dev(ys), dev(vs), dev([base]), dev([base]), dev([h]), xo, yo)
        assert ctx.stats()["n_p2p"] > 0 and ctx.stats()["n_e2l"] == 0
    finally:
        ctx.close()
    for got, terms in ((host(xo), dx * f), (host(yo), dy * f)):
        # 12 roundings a term, n of the sum
        assert np.all(np.abs(got - terms.sum(1)) <= (n + 12) * 2.0 ** -52 * np.abs(terms).sum(1))
