"""The bound within which the one-launch purification trusts its quickly summed traces (CPU).

The quick sum and the sum in the defining order differ by at most a rounding per addition in the
longest chain of each. The chains grow with the order; the bound has to grow with them.
"""
import ctypes as C
import math

import pytest

from pm7b200 import api


def _slack(n):
    f = api.lib()._ZN3pm713sp2_sum_slackEi
    f.restype, f.argtypes = C.c_double, [C.c_int32]
    return f(n)


def _additions(n):
    t = math.ceil(n / 64)
    blocks = t * (t + 1) // 2
    quick = math.ceil(128 * blocks / (16 * 128)) + math.log2(16) + math.log2(32) + 8
    defined = 1 + 64 + math.ceil(blocks / 256) + math.log2(32) + 8
    return quick + defined


@pytest.mark.parametrize("n", [2, 121, 767, 2004, 6000, 9400, 9900, 12000, 20000, 40000])
def test_the_bound_covers_both_orders_of_summation(n):
    assert _slack(n) >= _additions(n) * 2.0 ** -53


@pytest.mark.parametrize("n", [2, 767, 6000, 9400])
def test_the_bound_is_what_it_was_where_it_holds(n):
    assert _slack(n) == 1.0e-13
