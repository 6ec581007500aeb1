"""Shards whose own size would take them to other forms than the unsplit solve (blocks per brick, cut
near-field segments, common far fields): force shards still assemble to the unsplit solve bit for bit,
potential shards to the roundings of their sums."""
import numpy as np
import pytest

import sharding
import treecodes as T
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("side,blocksize", [(23, 32), (46, 16)])   # 8464 bricks; shards of 1693
def test_force_shards_across_the_forms(side, blocksize, precision):
    w = W.lamb_oseen_force(n=200000, blocks_per_side=side, h=1.0 / (side * blocksize))
    args = [w[k] for k in ("theta", "xs", "ys", "vs", "x0s", "y0s", "hs")]
    assert (blocksize // 8) ** 2 * len(w["x0s"]) > 8192
    ctx = T.Context(device=0, precision=precision)
    try:
        ctx.set_blocksize(blocksize)
        xo, yo = ctx.force_mrag_host(*args)
        parts = [sharding.solve_shard(ctx, *args, r, 5) for r in range(5)]
        sx, sy = sharding.assemble(parts, len(w["x0s"]), blocksize)
        assert np.array_equal(sx, xo) and np.array_equal(sy, yo)
        # the setting ends with the shard: a lone solve is planned by its own size again
        idx = parts[0][0]
        ax, ay = ctx.force_mrag_host(*args[:4], *(w[k][idx] for k in ("x0s", "y0s", "hs")))
        ctx2 = T.Context(device=0, precision=precision)
        ctx2.set_blocksize(blocksize)
        bx, by = ctx2.force_mrag_host(*args[:4], *(w[k][idx] for k in ("x0s", "y0s", "hs")))
        ctx2.close()
        assert np.array_equal(ax, bx) and np.array_equal(ay, by)
        assert ctx.lib.tc_set_whole_blocks(ctx.h, -1) == 1   # TC_ERR_INVALID
    finally:
        ctx.close()


def test_potential_shards_to_roundings():
    r = np.random.default_rng(61)
    n, m = 20000, 270001   # the whole solve has common far fields, a fifth of it does not
    xs, ys, vs, xt, yt = r.random(n), r.random(n), r.standard_normal(n), r.random(m), r.random(m)
    ctx = T.Context(device=0)
    try:
        whole = ctx.potential_host(0.5, xs, ys, vs, xt, yt)
        parts = [sharding.solve_potential_shard(ctx, 0.5, xs, ys, vs, xt, yt, k, 5) for k in range(5)]
    finally:
        ctx.close()
    got = sharding.assemble_potential(parts, m)
    pick = r.integers(0, m, 200)
    scale = np.abs(0.5 * vs * np.log((xt[pick, None] - xs) ** 2 + (yt[pick, None] - ys) ** 2)).sum(1)
    # at most n + 32 additions in either order
    assert np.all(np.abs(got - whole)[pick] <= 2 * (n + 32) * 2.0 ** -53 * scale)
