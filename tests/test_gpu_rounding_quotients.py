"""Quotients through the uncorrected reciprocal of the straight-line maps
against the IEEE division where they lie next to rounding boundaries: the
numerators within three of the smallest distances a quotient can have from a
midpoint, for all divisors just below a power of two (where a reciprocal that is
not the nearest could show) and for random ones."""
import ctypes

import pytest

from elegant_b200 import _native as nat

pytestmark = pytest.mark.gpu


def test_quotients_next_to_midpoints():
    f = nat.load_library().b2e_selftest_quotient
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int64, ctypes.c_uint64, ctypes.POINTER(ctypes.c_int64)]
    n = (ctypes.c_int64 * 5)(*[-1] * 5)
    assert f(4_000_000_000, 5, n) == 0
    print("reciprocals that are not the nearest: near 2", n[1], "random", n[3])
    assert [n[0], n[2], n[4]] == [0, 0, 0]
    assert n[1] >= 0 and 0 <= n[3] < 4000
