"""GPU checks of the substitutions' hand-over in groups of 8 rows (marked gpu).

Every CTA waits for all groups of its copy of x before it leaves a pass, the
block solved last included, which no other block waits for; the ensemble's one
launch sets the same barriers up again for its second pass.  Sizes whose last
group or last block is narrow, whose blocks are fewer than the CTAs, and that give
a warp several blocks.  The ensemble's instances reproduce the single-system
engine, and a lone solve the oracle, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2, 6, 8, 10, 32, 34, 40, 66, 258, 322]


def test_ensemble_instances_equal_single_runs(pkg):
    cfg = [pkg.dconf.generate_internal(n, 11 + n)[:2] for n in SIZES]

    def data():
        sd = pkg.SimulationData()
        sd.precision, sd.step_count_limited, sd.step_count_limit = 1e-6, True, 5
        sd.external_stress = pkg.FixedRateProtocol(0.05, 0.0)
        return sd

    ens = pkg.Ensemble(data(), cfg)
    res = ens.run()
    for k, (x, y) in enumerate(cfg):
        sd = data()
        sd.set_positions(x, y)
        e = pkg.Engine(sd)
        r = e.run()
        assert (res[k].successful_steps, res[k].failed_steps) == (r.successful_steps,
                                                                  r.failed_steps), SIZES[k]
        assert np.array_equal(ens.positions(k)[0], e.positions()[0]), SIZES[k]
        e.close()
    ens.close()


@pytest.mark.parametrize("n", SIZES + [2114])
def test_solve_equal_to_oracle(pkg, restated, n):
    rng = np.random.default_rng(n)
    a = np.eye(n) + rng.uniform(-0.5, 0.5, (n, n)) / n
    x, y, _ = pkg.dconf.generate_internal(n, 3)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    e = pkg.Engine(sd)
    e.set_matrix(a)
    assert e.factor() == 0
    for g in rng.normal(size=(3, n)):
        assert np.array_equal(e.solve(g)[0], restated.lu_solve(a, g)[0])
    e.close()
