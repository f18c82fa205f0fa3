"""How the tensor-core batched sum splits a batch into CTAs of four and of two solves.

The choice looks at the last few waves only; here it is compared with the
choice over every split, and its cost must not grow with the batch.
"""
import time

import pytest

from entropydecreaseboltzmann_gb300._lib import lib

fours = lib._ZN3edb8tc_foursEiiii  # edb::tc_fours(S, N, C, sms)


def _every_split(S, N, C, sms):
    two = 0.67 if N <= 16 else 0.63

    def waves(groups):
        return -(-groups * N * C // sms)

    best, four = 1e30, S
    for g4 in range((S + 3) // 4, -1, -1):
        n4 = min(S, 4 * g4)
        n2 = S - n4
        t = waves(g4) + two * waves((n2 + 1) // 2)
        if n2 > 0 and n4 > 0:
            t = 1.03 * t + 0.02
        if t < best - 1e-9:
            best, four = t, n4
    return four


@pytest.mark.parametrize("N", [13, 14, 17, 18, 21, 23, 25, 27, 30, 31])
def test_the_last_waves_hold_the_best_split(N):
    sizes = list(range(1, 130)) + [200, 257, 333, 500, 777, 1024, 2999, 4096]
    for C in (1, 3, 4, 8, N):
        for S in sizes:
            for sms in (152, 132):
                assert fours(S, N, C, sms) == _every_split(S, N, C, sms), (S, C, sms)


def test_the_cost_does_not_grow_with_the_batch():
    t = []
    for S in (4096, 40_000_000):
        best = 1e30
        for _ in range(20):
            t0 = time.perf_counter()
            fours(S, 13, 1, 152)
            best = min(best, time.perf_counter() - t0)
        t.append(best)
    assert t[1] < 20 * t[0]
