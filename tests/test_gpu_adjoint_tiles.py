"""GPU check of the adjoint's pair sweeps at the edges of their tiles (marked gpu).

Sizes with a ragged last row tile and a ragged last column tile, on either side
of the size at which the column tiles widen.  The bounds are the ones the
adjoint is held to elsewhere: central differences (h = 1e-6) to 1e-5 relative,
and the adjoint against the tangent-linear derivative to 1e-10 relative.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [18, 130, 2048, 2050])
def test_pair_tiles(pkg, n):
    x, y, _ = pkg.dconf.generate_internal(n, 1003)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    sd.external_stress = pkg.FixedRateProtocol(0.08, 0.0)
    sd.calculate_strain_during_simulation = True
    e = pkg.Engine(sd)
    e.record_steps(True)
    e.advance(2)
    t0s, hs = e.recorded_steps()
    _, g, gt = e.adjoint(x, t0s, hs)
    dx = np.random.default_rng(n).standard_normal(n)
    _, d = e.tangent(x, t0s, hs, dx, 0.3)
    ad = float(g @ dx) + 0.3 * gt
    assert abs(ad - d) <= 1e-10 * (float(abs(g) @ abs(dx)) + abs(0.3 * gt))
    # the coordinate the strain depends on most in the first and the last row tile
    for lo in (0, (n - 1) // 128 * 128):
        i = lo + int(np.argmax(abs(g[lo:])))
        xp, xm = x.copy(), x.copy()
        xp[i] += 1e-6
        xm[i] -= 1e-6
        fd = (e.replay(xp, t0s, hs)[0] - e.replay(xm, t0s, hs)[0]) / 2e-6
        assert abs(fd - g[i]) <= 1e-5 * abs(g).max(), (i, fd, g[i])
