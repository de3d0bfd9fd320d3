"""GPU checks of factors that are not finite (marked gpu): the oracle skips every
update whose value is exactly 0, so an infinite or NaN factor beside it has no
effect, and the solutions are the oracle's.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def factor_solve(pkg, a, rhs):
    n = len(a)
    x, y, _ = pkg.dconf.generate_internal(n, 3)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    e = pkg.Engine(sd)
    e.set_matrix(a)
    e.factor()
    out = [e.solve(g)[0] for g in rhs]
    e.close()
    return out


@pytest.mark.parametrize("n", [4, 32, 34, 66, 322])
def test_overflowed_column(pkg, restated, n):
    """A finite matrix whose last column overflows in the elimination: the last
    unknown is 0 and the infinite entries above the diagonal have no effect."""
    a = np.tril(np.full((n, n), -0.25 / n), -1) + np.eye(n)
    a[1:, 0] = -1
    a[:, -1] = 1.5e308
    rhs = np.random.default_rng(n).normal(size=(2, n))
    for g, dx in zip(rhs, factor_solve(pkg, a, rhs)):
        want = restated.lu_solve(a, g)[0]
        assert np.isfinite(want).all() and want[-1] == 0
        assert np.array_equal(dx, want)


def test_overflowed_column_mixed(pkg):
    """The same in FP32 by the mixed form's pivoted LU (the largest float is 3.4e38), in
    one block (its trailing update, on the tensor cores, makes NaN of infinities):
    its solves skip the zero as well, so the solution stays finite."""
    n = 32
    a = np.tril(np.full((n, n), -0.25 / n), -1) + np.eye(n)
    a[1:, 0] = -1
    a[:, -1] = 2e38
    x, y, _ = pkg.dconf.generate_internal(n, 3)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    sd.precision_mode = pkg._lib.D4_PREC_MIXED
    e = pkg.Engine(sd)
    e.set_block_lu(False)
    e.set_matrix(a)
    e.factor()
    dx, _ = e.solve(np.ones(n))
    assert np.isfinite(dx).all()
    e.close()


@pytest.mark.parametrize("n,row,col", [(32, 5, 2), (32, 31, 30), (66, 5, 2), (130, 63, 40)])
def test_nan_multiplier_of_zeros(pkg, restated, n, row, col):
    """A NaN multiplier whose row of U, and whose unknown, are zeros: no effect in the
    block's own rows and in the columns right of it."""
    a = np.eye(n) + np.triu(np.full((n, n), 0.25), 1)
    a[col, col + 1:] = 0
    a[row, col] = np.nan
    g = np.random.default_rng(n).normal(size=n)
    g[col] = 0
    want = restated.lu_solve(a, g)[0]
    assert np.isfinite(want).all()
    assert np.array_equal(factor_solve(pkg, a, [g])[0], want)
