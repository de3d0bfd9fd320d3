"""GPU check of the block LU's pivots at the ends of the FP32 range (marked gpu): a
pivot above 2^126 or below 2^-126, whose reciprocal the Gauss-Jordan inverse does not
form, goes to the pivoted LU; the solution is right either way.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pivot", [2.0 ** 127, 1.5 * 2.0 ** 126, 2.0 ** -126, 2.0 ** -127])
@pytest.mark.parametrize("place", [0, 5, 130, 255])
def test_extreme_pivot(pkg, pivot, place):
    n = 256
    x, y, _ = pkg.dconf.generate_internal(n, 5)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    sd.precision_mode = pkg._lib.D4_PREC_MIXED
    e = pkg.Engine(sd)
    d = np.ones(n)
    d[place] = pivot
    g = np.random.default_rng(place).normal(size=n)
    g[place] *= pivot  # so that the solution is of order 1
    before = e.mixed_stats()
    e.set_matrix(np.diag(d))
    assert e.factor() == 0
    dx, _ = e.solve(g)
    after = e.mixed_stats()
    assert after["block_factorizations"] == before["block_factorizations"] + 1
    inside = 2.0 ** -126 <= pivot <= 2.0 ** 126
    assert after["fallbacks"] == before["fallbacks"] + (0 if inside else 1)
    # FP32's rounding of each entry: refinement stops at 1e-12 of the largest |g|
    want = g / d
    assert np.abs(np.delete(dx - want, place)).max() <= 1e-6
    if pivot > 1:
        assert abs(dx[place] - want[place]) <= 1e-6
    e.close()
