"""GPU checks of the device block that the pattern analysis keeps between calls
(marked gpu).
"""
import importlib

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
