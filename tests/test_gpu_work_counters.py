"""Work counters of a potential with common far fields: a cell on a set's common list is counted as
one translation, not as evaluated from its multipoles for each target."""
import numpy as np
import pytest

import treecodes as T
from tc_helpers import gpu_potential

pytestmark = pytest.mark.gpu


def test_every_accepted_cell_is_counted_once():
    r = np.random.default_rng(51)
    n, m = 50000, 1 << 18   # 8192 groups of 32: 2048 sets of 128
    w = dict(theta=0.5, xs=r.random(n), ys=r.random(n), vs=r.standard_normal(n), xt=r.random(m),
             yt=r.random(m))
    ctx = T.Context(device=0)
    try:
        gpu_potential(ctx, w)
        whole = ctx.stats()
        # no sets below 262,144 targets: every accepted (target, cell) pair is evaluated
        accepted = 0
        for lo in range(0, m, m // 2):
            part = dict(w, xt=w["xt"][lo:lo + m // 2], yt=w["yt"][lo:lo + m // 2])
            gpu_potential(ctx, part)
            st = ctx.stats()
            accepted += st["e2p_pairs"]
            assert st["e2l_pairs"] == 0 and st["n_e2l"] == 0 and st["l2p_targets"] == 0
        ctx.set_precision(1)   # nor in the mixed form
        gpu_potential(ctx, w)
        mixed = ctx.stats()
    finally:
        ctx.close()
    assert mixed["e2p_pairs"] == accepted and mixed["e2l_pairs"] == 0
    assert whole["e2l_pairs"] > 0 and whole["n_e2l"] == whole["e2l_pairs"]
    assert whole["l2p_targets"] == m
    assert whole["e2p_pairs"] + 128 * whole["e2l_pairs"] == accepted
