"""The sweeps' division by a divisor known ahead (csrc/sweep.cuh) is the correctly
rounded one, bit for bit."""
import ctypes
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(3))
def test_quotients(cuda, seed):
    here = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cuda")
    subprocess.run(["make", "-C", here, "divide.so"], check=True, capture_output=True)
    lib = ctypes.CDLL(os.path.join(here, "divide.so"))
    bad, first = ctypes.c_ulonglong(), (ctypes.c_double * 2)()
    n = 200_000_000
    assert lib.compare_division(ctypes.c_ulonglong(seed * n), ctypes.c_longlong(n), ctypes.byref(bad), first) == 0
    assert bad.value == 0, [v.hex() for v in first]
