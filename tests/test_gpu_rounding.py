"""The reciprocals, quotients and square roots of the straight-line element
maps against the IEEE operators, bit for bit: random significands over 60
binades, operands around 1 and around powers of two, exact quotients and
squares, and operands placed next to rounding boundaries."""
import ctypes

import pytest

from elegant_b200 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [1, 77])
def test_shared_iterations_round_as_the_ieee_operators(seed):
    f = nat.load_library().b2e_selftest_rounding
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int64, ctypes.c_uint64, ctypes.POINTER(ctypes.c_int64)]
    bad = (ctypes.c_int64 * 4)(-1, -1, -1, -1)
    assert f(3_000_000_000, seed, bad) == 0
    assert list(bad) == [0, 0, 0, 0]
