"""GPU checks at the edges of the row and column splits (marked gpu).

GMRES: an attempt with the sparse solver against the same attempt with the dense
LU, for row counts that leave the last block few rows or none, and with more than
32 rows per block and more than 16 column chunks; bound as elsewhere 1e-12 in the
positions.  Mixed form: an attempt whose residual product has a ragged last chunk
of columns and block of rows against the FP64 form; bound as elsewhere 1e-10.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def attempt(pkg, n, h, **kw):
    x, y, _ = pkg.dconf.generate_internal(n, 1001)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    for k, v in kw.items():
        setattr(sd, k, v)
    e = pkg.Engine(sd)
    r, xb, xh, x2 = e.attempt(0.0, h)
    st = e.solver_stats() if "solver" in kw else None
    e.close()
    return (xb, xh, x2), st


@pytest.mark.parametrize("n,h", [(18, 1e-5), (34, 1e-5), (130, 1e-5), (514, 1e-6), (4810, 1e-7)])
def test_gmres_rows(pkg, n, h):
    kw = dict(cutoff_multiplier=3.2, heaviside_cutoff=True)
    got, st = attempt(pkg, n, h, solver=pkg._lib.D4_SOLVER_GMRES, **kw)
    want, _ = attempt(pkg, n, h, **kw)
    assert st["solves"] == 6 and st["fallbacks"] == 0
    for a, b in zip(got, want):
        assert np.abs(a - b).max() < 1e-12


@pytest.mark.parametrize("n", [2050, 2314])
def test_mixed_rows(pkg, n):
    got, _ = attempt(pkg, n, 1e-7, precision_mode=pkg._lib.D4_PREC_MIXED)
    want, _ = attempt(pkg, n, 1e-7)
    for a, b in zip(got, want):
        assert np.abs(a - b).max() < 1e-10
