"""GPU checks that contexts of different sizes do not disturb one another (marked
gpu).  The shared-memory limit of a kernel is the process's, not the context's, so
it may not follow the size of the context that was created, or launched, last.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ensemble(pkg, sizes):
    sd = pkg.SimulationData()
    sd.precision, sd.step_count_limited, sd.step_count_limit = 1e-6, True, 3
    sd.external_stress = pkg.FixedRateProtocol(0.05, 0.0)
    return pkg.Ensemble(sd, [pkg.dconf.generate_internal(n, n)[:2] for n in sizes])


def test_small_ensemble_beside_a_large_one(pkg):
    alone = ensemble(pkg, [322, 128])
    alone.run()
    want = alone.positions(0)[0]
    alone.close()
    large = ensemble(pkg, [322, 128])
    small = ensemble(pkg, [64])
    large.run()
    small.run()
    assert np.array_equal(large.positions(0)[0], want)
    small.close()
    large.close()

def test_gmres_contexts_on_two_threads(pkg):
    """Two contexts whose GMRES takes different numbers of rows per CTA (20 and 32)."""
    import threading

    errors = []

    def steps(n):
        x, y, _ = pkg.dconf.generate_internal(n, n)
        sd = pkg.SimulationData()
        sd.set_positions(x, y)
        sd.cutoff_multiplier, sd.heaviside_cutoff = 3.2, True
        sd.solver = pkg._lib.D4_SOLVER_GMRES
        e = pkg.Engine(sd)
        try:
            want = e.attempt(0.0, 1e-5)[1]
            for _ in range(400):
                assert np.array_equal(e.attempt(0.0, 1e-5)[1], want)
        except Exception as err:
            errors.append((n, err))
        e.close()

    threads = [threading.Thread(target=steps, args=(n,)) for n in (40, 64)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
