"""Bodies of an ensemble that coincide, exactly or in the FP32 coordinates the force loop stages, merge as in
the oracle's FP64 scan: within a fold of 64 bodies, across folds, and as a whole system."""
import numpy as np
import pytest

from gregpackagescpp_b200.ensemble import Ensemble
from gregpackagescpp_b200.ics import AU, ensemble
from test_ensemble_gpu import DT, oracle_run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies", [1, 2, 4])
@pytest.mark.parametrize("n,pairs", [(2, [(0, 1)]), (3, [(0, 2)]), (40, [(3, 17), (20, 21)]), (64, [(0, 63)]),
                                     (130, [(1, 2), (5, 70), (64, 127), (128, 129)])])
@pytest.mark.parametrize("apart", [0.0, 1.0e3])
def test_coincident_bodies_merge(gpu, oracle, n, pairs, apart, bodies):
    """`apart` metres: below the 10 to 20 km that FP32 resolves in a system of 1 AU, and below the radii."""
    m, r, x, v = ensemble(1, 500 + n, n_min=n, n_max=n, r_ball=1.0 * AU)[1:]
    r = np.full(n, 1.0e4)
    for i, j in pairs:
        x[j] = x[i] + np.array([apart, 0.0, 0.0])
    e = Ensemble(np.array([0, n]), m, x, v, r, merge=True, dt=DT)
    e.set_threads(128)
    e.set_bodies_per_thread(bodies)
    e.evolve(2)
    counts, merges, _ = e.counts()
    rows = np.concatenate([m[:, None], r[:, None], np.ones((n, 1)), x, v, np.zeros((n, 3))], 1)
    rows = oracle.merge_overlapping(rows)
    mo, ro, xo, vo = oracle_run(oracle, rows[:, 0].copy(), rows[:, 1].copy(), rows[:, 2].copy(), rows[:, 3:6].copy(),
                                rows[:, 6:9].copy(), 2, True)
    assert merges == len(pairs) and counts[0] == len(mo) == n - len(pairs)
    st = e.state()[0]
    np.testing.assert_allclose(st["m"], mo, rtol=1e-15)
    np.testing.assert_allclose(st["r"], ro, rtol=1e-14)
    assert np.abs(st["x"] - xo).max() <= 1e-9 * np.abs(xo).max()
    assert np.abs(st["v"] - vo).max() <= 1e-7 * np.abs(vo).max()
