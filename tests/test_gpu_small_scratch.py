"""Small solves take no memory from the pool once their buffers have grown: the list build's scratch
runs lie in the sort's record buffer, as in larger solves."""
import ctypes

import numpy as np
import pytest

import treecodes as T
from tc_helpers import dev, dev_empty

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8   # CU_MEMPOOL_ATTR_USED_MEM_CURRENT, _HIGH


class Pool:
    """The device's default memory pool, which the library's buffers come from."""

    def __init__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.pool = ctypes.c_void_p()
        assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), 0) == 0

    def get(self, attr):
        v = ctypes.c_uint64()
        assert self.cu.cuMemPoolGetAttribute(self.pool, attr, ctypes.byref(v)) == 0
        return v.value

    def reset_high(self):
        v = ctypes.c_uint64(0)
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_HIGH, ctypes.byref(v)) == 0


@pytest.mark.parametrize("n", [3000, 4096, 16384])
@pytest.mark.parametrize("kind", ["force", "potential"])
def test_repeated_small_solves_allocate_nothing(kind, n):
    r = np.random.default_rng(71)
    xs, ys, vs = dev(r.random(n)), dev(r.random(n)), dev(r.standard_normal(n))
    out = [dev_empty(1024), dev_empty(1024)]
    ctx = T.Context(device=0)
    try:
        def solve():
            if kind == "force":
                ctx.force_mrag_device(0.5, xs, ys, vs, dev([0.25]), dev([0.25]), dev([1 / 64]), *out)
            else:
                ctx.potential_device(0.5, xs, ys, vs, xs[:1024], ys[:1024], out[0])
        for _ in range(3):   # buffers and list regions reach their sizes
            solve()
        pool = Pool()
        pool.reset_high()
        before = pool.get(USED_CURRENT)
        solve()
        assert pool.get(USED_HIGH) == before
    finally:
        ctx.close()
