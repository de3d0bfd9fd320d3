"""GPU checks of the FP64 LU (d4_lu_exact.cuh) at the sizes and values where its
paths change (marked gpu): one block, a narrow last block, one row or column
group, each tile shape of the trailing update (64 x 32, 64 x 64, 128 x 64 from
about n = 1900), passes repeated after a swap, and values that leave the fast
quotients (outside the window |v| in [2^-400, 2^401), pivots whose significand
is all ones).  The factors keep the oracle's operation order, so the solutions
are equal to the oracle's in every case.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dominant(n, rng):
    a = rng.uniform(-0.5, 0.5, (n, n)) / n
    a[np.arange(n), np.arange(n)] = 1 + rng.uniform(0, 0.5, n)
    return a


def swapped(n, rng):
    """Two row exchanges inside blocks and two across them."""
    a = dominant(n, rng)
    for i, j in ((0, 1), (n // 3, n // 3 + 1), (n // 4, n - 1), (n // 2, (n // 2 + 40) % n)):
        a[[i, j]] = a[[j, i]]
    return a


def window(n, rng):
    """Every fifth column scaled below the quotient window (its multipliers stay
    ordinary), every seventh above it."""
    a = dominant(n, rng)
    a[:, ::5] *= 2.0 ** -500
    a[:, 3::7] *= 2.0 ** 450
    return a


def all_ones(n, rng):
    """Unit upper triangle, so every pivot is the largest double below 1."""
    a = np.tril(rng.uniform(-0.5, 0.5, (n, n)), -1)
    a[np.arange(n), np.arange(n)] = np.nextafter(1.0, 0.0)
    return a


CASES = [(dominant, n) for n in (2, 30, 32, 34, 64, 66, 130, 258, 642, 1026, 2050)]
CASES += [(swapped, n) for n in (34, 66, 130, 386, 1026)]
CASES += [(window, n) for n in (34, 130, 386)] + [(all_ones, n) for n in (34, 130, 386)]


@pytest.mark.parametrize("make,n", CASES, ids=lambda v: v.__name__ if callable(v) else str(v))
def test_factor_solve_equal_to_oracle(pkg, restated, make, n):
    rng = np.random.default_rng(n)
    a = make(n, rng)
    g = rng.normal(size=n)
    x, y, _ = pkg.dconf.generate_internal(n, 3)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    e = pkg.Engine(sd)
    e.set_matrix(a)
    assert e.factor() == 0
    dx, _ = e.solve(g)
    dx_o, sing, piv = restated.lu_solve(a, g)
    assert sing == 0
    assert np.array_equal(dx, dx_o)
    swaps = int((piv != np.arange(n)).sum())
    st = e.lu_stats()
    assert (st["swaps"], st["passes"]) == (swaps, -(-n // 32) + swaps)
    e.close()
