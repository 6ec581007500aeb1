"""Leaf moments, bit for bit, against a restatement of the four strided sums in NumPy: leaves of
one source to the cap, around the kernels' batches of 128 sources and four chains, leaves without
weight, and a tree of more nodes than the warp-per-node form takes."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "2d-treecodes_b200"))

pytestmark = pytest.mark.gpu


def leaf_moments(x, y, v):
    w = np.abs(v)
    total = []
    lanes = []
    for q in range(4):   # cumsum adds one term after another
        lanes.append([np.cumsum(a[q::4])[-1] if len(a[q::4]) else 0.0 for a in (v, w, x * w, y * w)])
    for k in range(4):
        total.append((lanes[0][k] + lanes[1][k]) + (lanes[2][k] + lanes[3][k]))
    r2 = 0.0
    for q in range(4):
        on = lanes[q][1] != 0
        cx, cy = (total[2] / total[1], total[3] / total[1]) if on else (0.0, 0.0)
        dx, dy = x[q::4] - cx, y[q::4] - cy
        if len(dx):
            r2 = max(r2, (dx * dx + dy * dy).max())
    return total, np.sqrt(r2)


@pytest.mark.parametrize("kind,n", [("potential", n) for n in
                                    (1, 2, 3, 4, 5, 31, 33, 127, 128, 129, 131, 255, 257, 511, 512,
                                     3001, 70001)] +
                                   [("force", n) for n in (1, 127, 129, 192, 20003, 6000001)])
def test_leaf_moments(kind, n):
    import torch
    import treecodes as T

    r = np.random.default_rng(n)
    x, y, v = r.random(n), r.random(n), r.uniform(-1, 1, n)
    v[:n // 5] = 0.0            # sources without weight, and chains and leaves of them
    x[:n // 5] *= 0.25
    y[:n // 5] *= 0.25
    d = [torch.tensor(a, device="cuda") for a in (x, y, v)]
    torch.cuda.synchronize()
    t = T.Context().tree(kind, *d)
    leaves = np.flatnonzero(t["inner"] == 0)
    assert (len(t["inner"]) >= 65536) == (n > 1000000)
    for i in leaves[::max(1, len(leaves) // 4000)]:
        s, e = t["s"][i], t["e"][i]
        if e == s:
            continue
        total, radius = leaf_moments(t["xs"][s:e], t["ys"][s:e], t["vs"][s:e])
        assert t["mass"][i] == total[0], (i, e - s)
        if total[1] != 0:
            assert t["xcom"][i] == total[2] / total[1] and t["ycom"][i] == total[3] / total[1], (i, e - s)
        assert t["r"][i] == radius, (i, e - s)
