"""GPU check of the pair tiles' field (f64::pair) against the general evaluation
(Field.eval, f64::xy) at the distances where its branches change (marked gpu):
the Taylor branch's edge, dx = 0 and dx so small that the quotients would leave
the normal range (the general evaluation's own path), the cell's half width, and
ordinary distances.  Both form every operation in the reference's order and
every quotient correctly rounded, so the stress is the same number.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DISTANCES = [(0.0, 0.25), (1e-200, 0.3), (-3e-120, 0.01), (1e-80, -0.2), (6e-4, 7e-4),
             (7e-4, 7.2e-4), (9.99e-4, 0.0), (1.01e-3, 0.0), (-2e-5, 3e-5), (0.4999, 0.4999),
             (-0.5, 0.1), (0.25, -0.5), (-0.123, 0.0456), (0.31, -0.27)]


@pytest.mark.parametrize("dx,dy", DISTANCES)
def test_pair_equals_general_field(pkg, dx, dy):
    # the second dislocation at the origin: the difference is dx, dy itself
    x, y = np.array([dx, 0.0]), np.array([dy, 0.0])
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    e = pkg.Engine(sd)
    v, _ = e.speeds(x, y, 0.0)
    f = pkg.Field().eval(np.array([dx]), np.array([dy]))[0][0]
    assert v[0] == -f and v[1] == f  # opposite signs: b_0 b_1 = -1
    va, _, _, _, _ = e.jacobian(x, y, 1e-6, 0.0, 1e-6)
    assert np.array_equal(va, v)  # the fused sweep's stress is the stress sweep's
    e.close()
