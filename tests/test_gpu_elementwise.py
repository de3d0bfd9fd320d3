"""GPU check of the row scaling and the half step's rescale at the edges of their
blocks of 256 rows and 8 columns (marked gpu): one attempt, whose second small step
solves with the rescaled matrix, against the oracle's, to the bound that attempts
are held to elsewhere (1e-12 in the positions)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [6, 18, 254, 258, 518])
def test_attempt_at_block_edges(pkg, restated, n):
    x, y, _ = pkg.dconf.generate_internal(n, 1001)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    e = pkg.Engine(sd)
    _, xb, xh, x2 = e.attempt(0.0, 1e-6)
    p = restated.params()
    mps, _, _, _ = restated.derived(p, n)
    xbo, xho, x2o, _, _, _ = restated.attempt(x, y, 0.0, 1e-6, p, np.full(n, mps))
    for a, b in ((xb, xbo), (xh, xho), (x2, x2o)):
        assert np.abs(a - b).max() < 1e-12
