"""Evaluation tasks: few target groups or bricks are cut into more tasks than many are.  The same
targets must give the same values whether they are solved alone (cut segments) or as part of a
large set (whole segments).  Only FP64 sums are regrouped: about 1e4 terms, so 1e4 * 2^-53."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "2d-treecodes_b200"))

pytestmark = pytest.mark.gpu
TOL = 1e4 * 2.0 ** -53


def rel(a, b):
    return float((a - b).norm() / b.norm())


def clustered(n, seed):
    r = np.random.default_rng(seed)
    x = np.where(r.random(n) < 0.5, r.random(n), 0.3 + 0.003 * r.standard_normal(n))
    y = np.where(r.random(n) < 0.5, r.random(n), 0.7 + 0.003 * r.standard_normal(n))
    return x, y, r.uniform(-1, 1, n)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("m", [1, 33, 32 * 500, 32 * 16384 - 31, 32 * 16384 + 1])
def test_potential_of_a_subset_equals_the_whole(precision, m):
    import torch
    import treecodes as T

    d = lambda a: torch.tensor(a, device="cuda")
    xs, ys, vs = map(d, clustered(30011, 3))
    big = 32 * 32768 + 7
    # the subset is compact, so its groups of 32 are the same targets in both solves: a copy of
    # every target 32 times makes each group one point
    r = np.random.default_rng(5)
    px, py = r.random(big // 32 + 1), r.random(big // 32 + 1)
    xt, yt = d(np.repeat(px, 32)), d(np.repeat(py, 32))
    ctx = T.Context(precision=precision)
    whole, part = torch.empty_like(xt), torch.empty(m, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    ctx.potential_device(0.5, xs, ys, vs, xt, yt, whole)
    ctx.potential_device(0.5, xs, ys, vs, xt[:m].clone(), yt[:m].clone(), part)
    # mixed: the near field keeps whole segments, FP32 rounding of the group's offsets aside
    assert rel(part, whole[:m]) < (TOL if precision == 0 else 1e-6)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("side", [1, 2, 5, 31, 33])
def test_force_of_a_subset_equals_the_whole(precision, side):
    import torch
    import treecodes as T
    import workloads as W

    d = lambda a: torch.tensor(a, device="cuda")
    xs, ys, vs = map(d, clustered(30011, 4))
    x0, y0, h = map(d, W.mrag_grid(48, 1.0 / (32 * 48)))   # 36,864 bricks: whole segments
    nb = side * side
    ctx = T.Context(precision=precision)
    whole = [torch.empty(1024 * len(x0), device="cuda", dtype=torch.float64) for _ in range(2)]
    part = [torch.empty(1024 * nb, device="cuda", dtype=torch.float64) for _ in range(2)]
    torch.cuda.synchronize()
    ctx.force_mrag_device(0.5, xs, ys, vs, x0, y0, h, *whole)
    ctx.force_mrag_device(0.5, xs, ys, vs, x0[:nb].clone(), y0[:nb].clone(), h[:nb].clone(), *part)
    # (the mixed form's tiles and FP32 sums are the same; its compensated sums add in FP64)
    for a, b in zip(part, whole):
        assert rel(a, b[:1024 * nb]) < (TOL if precision == 0 else 1e-9)


@pytest.mark.parametrize("theta,order", [(0.3, 12), (0.5, 12), (0.7, 8), (0.5, 28), (1.0, 4)])
def test_common_far_fields_equal_the_groups_own(theta, order):
    """FP64 targets enough for sets with a common far field (262,144) against the same targets in
    solves too small for them: spread and clustered, some of them far outside the sources, some
    coincident (sets of one point), and one at infinity, which must not reach its neighbours.  The
    local expansions leave out 1e-17 of a cell's weight; FP64 sums are regrouped."""
    import torch
    import treecodes as T

    d = lambda a: torch.tensor(a, device="cuda")
    xs, ys, vs = map(d, clustered(30011, 6))
    r = np.random.default_rng(9)
    m = 270001
    x, y, _ = clustered(m, 10)
    x[:20000] = 3 * x[:20000] - 1
    x[20000:20200] = x[20000]
    y[20000:20200] = y[20000]
    x[30000] = np.inf
    p = r.permutation(m)
    xt, yt = d(x[p]), d(y[p])
    ctx = T.Context()
    ctx.set_orders(potential_order=order)
    whole = torch.empty(m, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    ctx.potential_device(theta, xs, ys, vs, xt, yt, whole)
    part = torch.empty_like(whole)
    for a in range(0, m, 90000):
        o = torch.empty(min(90000, m - a), device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        ctx.potential_device(theta, xs, ys, vs, xt[a:a + 90000].clone(), yt[a:a + 90000].clone(), o)
        part[a:a + 90000] = o
    fin = torch.isfinite(xt)
    assert bool(torch.isfinite(whole[fin]).all())
    assert rel(whole[fin], part[fin]) < TOL
