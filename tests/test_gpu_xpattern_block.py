"""GPU checks of the device block that the pattern analysis keeps between calls
(marked gpu).
"""
import importlib
import os
import subprocess
import sys

import numpy as np
import pytest

xp = importlib.import_module("2d4_b200.xpattern")
pytestmark = pytest.mark.gpu


def configuration(n=1000):
    rng = np.random.default_rng(n)
    return rng.uniform(-0.5, 0.5, n), rng.uniform(-0.5, 0.5, n), np.sign(rng.uniform(-1, 1, n))


def test_a_small_call_keeps_the_large_block(pkg):
    lib = pkg._lib.load()
    c = configuration()
    xp.direct_fourier(*c, 1024)
    before = lib.d4_device_allocations()
    xp.direct_fourier(*c, 64)
    xp.direct_fourier(*c, 1024)
    assert lib.d4_device_allocations() == before


RESET = """
import ctypes, importlib, sys
import numpy as np
sys.path.insert(0, %r)
pkg = importlib.import_module("2d4_b200")
xp = importlib.import_module("2d4_b200.xpattern")
rng = np.random.default_rng(1)
c = rng.uniform(-0.5, 0.5, 500), rng.uniform(-0.5, 0.5, 500), np.sign(rng.uniform(-1, 1, 500))
want = xp.direct_fourier(*c, 256)
lib = pkg._lib.load()
before = lib.d4_device_allocations()
cudart = ctypes.CDLL("libcudart.so.12")  # the one that the library has loaded
assert cudart.cudaDeviceReset() == 0
p = ctypes.c_void_p()  # the runtime hands the same addresses out again
assert cudart.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(8 << 20)) == 0
assert cudart.cudaMemset(p, 7, ctypes.c_size_t(8 << 20)) == 0
assert np.array_equal(xp.direct_fourier(*c, 256), want)
assert lib.d4_device_allocations() == before + 1  # not the block of before the reset
got = np.zeros(8 << 20, np.uint8)
assert cudart.cudaMemcpy(got.ctypes.data_as(ctypes.c_void_p), p, ctypes.c_size_t(8 << 20), 2) == 0
assert (got == 7).all()
"""


def test_device_reset_by_the_program():
    """A block of before a device reset is not used again, nor freed when its address
    has become another allocation's."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", RESET % root], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
