"""Cell ranges of the tree, for every node, against the sorted keys: child counts around the
probing distances of the eight-lane search (8, 64, 512), empty children, and a tree of more inner
cells than that search takes."""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "2d-treecodes_b200"))

pytestmark = pytest.mark.gpu

LMAX = 15


@pytest.mark.parametrize("counts", [(200, 0, 0, 0), (0, 0, 0, 193), (0, 8, 9, 200), (7, 0, 63, 200),
                                    (64, 65, 66, 9), (511, 512, 513, 1), (1, 4096, 8, 4097),
                                    (32768, 0, 1, 40000), (1500000,) * 4])
def test_every_range_is_its_keys(counts):
    import torch
    import treecodes as T

    r = np.random.default_rng(sum(counts))
    x = np.concatenate([r.random(c) * 0.5 + 0.5 * (q & 1) for q, c in enumerate(counts)])
    y = np.concatenate([r.random(c) * 0.5 + 0.5 * (q >> 1) for q, c in enumerate(counts)])
    d = [torch.tensor(a, device="cuda") for a in (x, y, np.ones(len(x)))]
    torch.cuda.synchronize()
    t = T.Context().tree("force", *d)
    keys = t["keys"].astype(np.int64)
    inner = t["child"] >= 0
    assert (inner.sum() > 16384) == (len(x) > 1000000)

    def spread(a):
        return sum(((a >> b) & 1) << (2 * b) for b in range(LMAX))

    level = t["level"].astype(np.int64)
    prefix = spread(t["cx"].astype(np.int64)) | spread(t["cy"].astype(np.int64)) << 1
    shift = 2 * (LMAX - level)
    assert np.array_equal(t["s"], np.searchsorted(keys, prefix << shift))
    assert np.array_equal(t["e"], np.searchsorted(keys, (prefix + 1) << shift))
    assert np.array_equal(t["e"] - t["s"], t["count"])
    assert np.array_equal(inner, (t["count"] > 192) & (level < LMAX))
