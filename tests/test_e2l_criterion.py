"""The force traversal's E2L test (classify in force.cu) decides on squares where it safely can.  The
rule, restated in IEEE double arithmetic, agrees with the reference's dist / r - 1 > 1 / theta
(drivers/treecode-force.cpp:136-141) on random and on borderline distances, and on the extremes
of r, d and theta."""
import numpy as np
import pytest


def exact(d2, r, inv_theta):
    with np.errstate(all="ignore"):
        return np.sqrt(d2) / r - 1.0 > inv_theta


def on_squares(d2, r, inv_theta):
    with np.errstate(all="ignore"):
        t = r * (1.0 + inv_theta)
        t2 = t * t
        yes = (t > 1e-140) & (d2 > t2 * (1.0 + 1e-12))
        no = (t > 1e-140) & (d2 < t2 * (1.0 - 1e-12))
        return np.where(yes, True, np.where(no, False, exact(d2, r, inv_theta))), yes | no


@pytest.mark.parametrize("theta", [0.05, 0.2, 0.3, 0.5, 0.7, 1.0, 3.0, 1e3, 1e-3])
def test_same_decisions(theta):
    g = np.random.default_rng(17)
    inv = 1.0 / theta
    r = np.exp(g.uniform(np.log(1e-8), np.log(10.0), 200000))
    d = np.exp(g.uniform(np.log(1e-8), np.log(1e3), 200000))
    # half of them around the border, down to an ulp off it
    k = r.size // 2
    d[:k] = r[:k] * (1.0 + inv) * (1.0 + g.choice([-1, 1], k) * 10.0 ** g.uniform(-17, -3, k))
    got, short = on_squares(d * d, r, inv)
    assert np.array_equal(got, exact(d * d, r, inv))
    assert short.mean() > 0.6   # the shortcut does decide most


def test_extremes():
    v = np.array([0.0, 5e-324, 1e-310, 1e-200, 1e-160, 1e-140, 1e-70, 1.0, 1e70, 1e140, 1e160, 1e200,
                  1e308, np.inf, np.nan])
    d, r = (a.ravel() for a in np.meshgrid(v, v))
    with np.errstate(all="ignore"):
        d2 = d * d
    for inv in [0.0, 1.0, 2.0, 1e8, np.inf, -0.5, -1.0, -2.0, -3.0, -np.inf, np.nan]:
        got, _ = on_squares(d2, r, inv)
        assert np.array_equal(got, exact(d2, r, inv)), inv
