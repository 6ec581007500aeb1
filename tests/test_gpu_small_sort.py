"""Sources and targets sorted in one block (up to 16,384): the same keys, permutation and sorted
sources as the allocation-free entry point's multi-launch sort of the same input, bit for bit, at
the edges of the block's item counts, with ties; and the host path's late values."""
import ctypes
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "2d-treecodes_b200"))

pytestmark = pytest.mark.gpu


def inputs(n, seed):
    r = np.random.default_rng(seed)
    x, y = r.random(n), r.random(n)
    x[n // 3:n // 2] = x[n // 3]   # equal keys keep their input order
    y[n // 3:n // 2] = y[n // 3]
    return x, y, r.uniform(-1, 1, n)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 1023, 1025, 4095, 4096, 4097, 16383, 16384, 16385])
def test_small_sort_equals_the_general_sort(n):
    import torch
    import treecodes as T

    x, y, v = inputs(n, n)
    dx, dy, dv = (torch.tensor(a, device="cuda") for a in (x, y, v))
    ctx = T.Context()
    torch.cuda.synchronize()
    t = ctx.tree("force", dx, dy, dv)
    keys, perm = (torch.empty(n, device="cuda", dtype=torch.int32) for _ in range(2))
    xs, ys, vs = (torch.empty(n, device="cuda", dtype=torch.float64) for _ in range(3))
    frame = torch.empty(4, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    rc = T.load().tc_sort_sources_noalloc(dx.data_ptr(), dy.data_ptr(), dv.data_ptr(), n,
                                          keys.data_ptr(), perm.data_ptr(), xs.data_ptr(),
                                          ys.data_ptr(), vs.data_ptr(), frame.data_ptr(),
                                          ctypes.c_void_p(None))
    assert rc == 0, T.last_error()
    for name, a in (("keys", keys), ("perm", perm), ("xs", xs), ("ys", ys), ("vs", vs)):
        assert np.array_equal(t[name], a.cpu().numpy()), name
    assert np.array_equal(t["frame"], frame[:3].cpu().numpy())


@pytest.mark.parametrize("m", [1, 32, 4096, 4097, 16384, 16385])
def test_small_solves_host_and_device_agree(m):
    import torch
    import treecodes as T

    x, y, v = inputs(5000, 7)
    tx, ty, _ = inputs(m, 8)
    tx = 1.5 * tx - 0.25   # targets outside the sources' frame too
    host = T.Context().potential_host(0.5, x, y, v, tx, ty)
    d = [torch.tensor(a, device="cuda") for a in (x, y, v, tx, ty)]
    out = torch.empty(m, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    T.Context().potential_device(0.5, *d, out)
    assert np.array_equal(out.cpu().numpy(), host)
    # against the direct sum: the truncation of order 12 at theta 0.5
    ref = torch.empty_like(out)
    T.Context().direct_potential_device(*d, ref)
    assert float((out - ref).norm()) < 1e-5 * float(ref.norm())


@pytest.mark.parametrize("n", [1, 4096, 4097, 16384, 16385])
def test_sources_and_targets_sorted_side_by_side(n):
    """One context, the targets' count moving between the forms (with the sources, by themselves,
    general): every target's value, against the direct sum (order 12 at theta 0.5, as above)."""
    import torch
    import treecodes as T

    x, y, v = inputs(n, n)
    d = [torch.tensor(a, device="cuda") for a in (x, y, v)]
    ctx = T.Context()
    for m in (1, 4096, 16385, 4097, 16384, 32769, 33):
        tx, ty, _ = inputs(m, m + 1)
        t = [torch.tensor(1.5 * a - 0.25, device="cuda") for a in (tx, ty)]
        out, ref = (torch.full((m,), float("nan"), device="cuda", dtype=torch.float64)
                    for _ in range(2))
        torch.cuda.synchronize()
        ctx.potential_device(0.5, *d, *t, out)
        T.Context().direct_potential_device(*d, *t, ref)
        assert float((out - ref).norm()) < 1e-5 * float(ref.norm()), m


@pytest.mark.parametrize("n", [16385, 18431, 18432, 18433, 1048577, 1572863, 1572864, 1572865,
                               1575936, 1575937])
def test_general_sort_is_stable_at_the_tiles_edges(n):
    """Both tile sizes of the radix passes, around whole tiles and the size where they change."""
    import torch
    import treecodes as T

    x, y, v = inputs(n, n)
    d = [torch.tensor(a, device="cuda") for a in (x, y, v)]
    torch.cuda.synchronize()
    t = T.Context().tree("potential", *d)
    assert np.array_equal(np.sort(t["perm"]), np.arange(n))
    keys = np.empty(n, t["keys"].dtype)
    keys[t["perm"]] = t["keys"]
    assert np.array_equal(t["perm"], np.argsort(keys, kind="stable"))
    for name, a in (("xs", x), ("ys", y), ("vs", v)):
        assert np.array_equal(t[name], a[t["perm"]]), name
