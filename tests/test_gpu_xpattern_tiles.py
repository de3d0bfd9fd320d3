"""GPU check of the pattern analysis at the edges of its tiles (marked gpu).

K = res/2 + 1 wave numbers below one tile, a whole number of tiles, the
remainders that thin tiles cover (1 to 16) and the first that they do not, and
numbers of dislocations around the staged chunk and its slices, with all, none
and some of them positive.  The bound is the one the analysis is held to
elsewhere: 1e-11 of the largest value.
"""
import importlib

import numpy as np
import pytest

import xpattern_ref

xp = importlib.import_module("2d4_b200.xpattern")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [2, 63, 64, 65, 80, 81, 129, 208])
@pytest.mark.parametrize("n,positive", [(1, 1), (17, 0), (33, 33), (300, 131), (1030, 515)])
def test_tiles(k, n, positive):
    rng = np.random.default_rng(100 * k + n)
    x, y = rng.uniform(-0.5, 0.5, n), rng.uniform(-0.5, 0.5, n)
    b = np.where(np.arange(n) < positive, 1.0, -1.0)
    rng.shuffle(b)
    res = 2 * (k - 1)
    got, want = xp.direct_fourier(x, y, b, res), xpattern_ref.direct_fourier(x, y, b, res)
    assert np.abs(got - want).max() <= 1e-11 * np.abs(want).max()
    assert np.array_equal(got, xp.direct_fourier(x, y, b, res))
