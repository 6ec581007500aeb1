"""The binomial table of the expansions (tc_math.cuh), restated: Pascal's triangle summed in double is
exact in every entry that a translation reads, those above 2^53 included."""
import math


def test_every_entry_used_is_exact():
    n = 64
    t = [[0.0] * n for _ in range(n)]
    for i in range(n):
        t[i][0] = 1.0
        for k in range(1, i + 1):
            t[i][k] = t[i - 1][k - 1] + (t[i - 1][k] if k < i else 0.0)
    for order in (4, 8, 12, 16, 20, 24, 28):
        for k in range(1, order + 1):
            # l up to the order in E2L and E2E, up to 31 in the sets' local expansions
            for l in range(1, max(order, 31) + 1):
                assert t[l + k - 1][k - 1] == math.comb(l + k - 1, k - 1)
