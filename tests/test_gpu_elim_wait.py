"""A wait of the FP64 LU's elimination that gives up is reported (marked gpu): the
self-test's column barriers lack an arrival, so the warps to the right wait until
their limit; the context stays usable.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_elimination_wait_gives_up(pkg, restated):
    n = 64
    x, y, _ = pkg.dconf.generate_internal(n, 3)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    e = pkg.Engine(sd)
    assert e.lib.d4_wait_selftest(e.ctx, 2) == pkg._lib.D4_ERR_STATE
    assert b"gave up" in e.lib.d4_last_error(e.ctx)
    assert e.lib.d4_wait_selftest(e.ctx, 3) == pkg._lib.D4_ERR_ARG
    rng = np.random.default_rng(n)
    a, g = np.eye(n) + rng.uniform(-0.5, 0.5, (n, n)) / n, rng.normal(size=n)
    e.set_matrix(a)
    assert e.factor() == 0
    assert np.array_equal(e.solve(g)[0], restated.lu_solve(a, g)[0])
    e.close()
