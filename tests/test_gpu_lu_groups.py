"""GPU checks of the FP64 LU's groups of CTAs that the other tests do not form (marked
gpu): clusters of one and two CTAs (ensembles of many instances of about one size) and
of four, against single-system runs bit for bit; and the whole grid on a matrix so
large that its look-ahead CTA takes update tiles of its own (from about n = 2200),
against the oracle, without row exchanges and with.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [160, 80, 40])  # clusters of 1, 2 and 4 on 148 SMs
@pytest.mark.parametrize("sizes", [(126, 130, 128, 130), (318, 322, 320, 322)])
def test_ensemble_clusters(pkg, count, sizes):
    cfg = [pkg.dconf.generate_internal(sizes[k % 4], 100 + k)[:2] for k in range(count)]

    def data():
        sd = pkg.SimulationData()
        sd.precision, sd.step_count_limited, sd.step_count_limit = 1e-6, True, 2
        sd.external_stress = pkg.FixedRateProtocol(0.05, 0.0)
        return sd

    ens = pkg.Ensemble(data(), cfg)
    res = ens.run()
    for k in (0, 1, 2, count // 2 + 1, count - 1):
        sd = data()
        sd.set_positions(*cfg[k])
        e = pkg.Engine(sd)
        r = e.run()
        assert (res[k].successful_steps, res[k].failed_steps) == (r.successful_steps,
                                                                  r.failed_steps), k
        assert np.array_equal(ens.positions(k)[0], e.positions()[0]), k
        e.close()
    ens.close()


@pytest.mark.parametrize("exchanges", [False, True])
def test_lookahead_takes_tiles(pkg, restated, exchanges):
    n = 2306  # a ragged last tile
    rng = np.random.default_rng(n)
    a = rng.uniform(-0.5, 0.5, (n, n)) / n
    a[np.arange(n), np.arange(n)] = 1 + rng.uniform(0, 0.5, n)
    if exchanges:
        for i, j in ((0, 1), (n // 4, n - 1)):
            a[[i, j]] = a[[j, i]]
    g = rng.normal(size=n)
    x, y, _ = pkg.dconf.generate_internal(n, 3)
    sd = pkg.SimulationData()
    sd.set_positions(x, y)
    e = pkg.Engine(sd)
    e.set_matrix(a)
    assert e.factor() == 0
    assert np.array_equal(e.solve(g)[0], restated.lu_solve(a, g)[0])
    e.close()
