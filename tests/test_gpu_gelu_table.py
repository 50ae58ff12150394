"""The table of GELU' at BF16 values holds the floats that the formula gives on
the device, bit for bit, for every BF16 value below 8 in magnitude, and tells the
others (and NaN) apart."""
import ctypes

import pytest

from elegant_b200 import _native as nat

pytestmark = pytest.mark.gpu


def test_every_bf16_value():
    f = nat.load_library().b2e_selftest_gelu_grad
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.POINTER(ctypes.c_int64)]
    bad = ctypes.c_int64(-1)
    assert f(ctypes.byref(bad)) == 0
    assert bad.value == 0
