"""The sample sort's plan, on the host: within the kernels' limits for every size, and with
so few buckets beyond their slots for records in random order that the fallback to digits
does not count (an overflow costs the attempt and up to 3 ms of digit passes)."""
import ctypes
import math

import pytest

from pauliprop import _lib

SIZES = sorted({4097, 5000, 2_200_000} | {int(4097 * 1.02 ** k) for k in range(318)}
               | {s + d for s in (549_450, 563_200, 614_400, 716_800, 900_000, 1_116_160, 1_331_200, 1_800_000, 2_000_000,
                                  2_199_000) for d in (-1, 0, 1)})


def plan(n):
    b, s, c = ctypes.c_int32(), ctypes.c_int32(), ctypes.c_int32()
    _lib.check(_lib.lib.pp_debug_sort_plan(n, ctypes.byref(b), ctypes.byref(s), ctypes.byref(c)))
    return b.value, s.value, c.value


def test_limits():
    for n in SIZES:
        b, s, c = plan(n)
        assert 1 < b <= 2048 and c in (2048, 4096) and b * s <= 16384 and b * s <= n
    assert plan(4096)[0] == 1 and plan(2_200_001)[0] == 0


@pytest.mark.parametrize("sizes", [SIZES[k::4] for k in range(4)])
def test_overflow_is_rare(sizes):
    for n in sizes:
        b, s, c = plan(n)
        # a bucket is the sum of s spacings of b * s random samples among n records, close to
        # n / b times a Gamma(s) variable over s; the chance that it is beyond c
        x = s * c / (n / b)
        tail = math.exp(-x) * sum(x ** k / math.factorial(k) for k in range(s))
        assert b * tail <= 1e-3, (n, b, s, c, b * tail)
