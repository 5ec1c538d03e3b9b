"""The ensemble's row chunks: systems of one chunk, of several, and of exactly a chunk give the
trajectories of any other chunking, merges included, and evolves may be cut anywhere."""
import numpy as np
import pytest

from gregpackagescpp_b200.ensemble import Ensemble
from gregpackagescpp_b200.ics import AU, ensemble

pytestmark = pytest.mark.gpu


def _systems(sizes, inflate):
    parts = [ensemble(1, 90 + k, n_min=n, n_max=n, r_ball=2.0 * AU)[1:] for k, n in enumerate(sizes)]
    m, r, x, v = (np.concatenate(a) for a in zip(*parts))
    return np.concatenate([[0], np.cumsum(sizes)]), m, r * inflate, x, v


@pytest.mark.parametrize("inflate", [1.0, 20.0])
def test_chunks_do_not_change_the_result(gpu, inflate):
    """Bit for bit: a row's sum does not depend on the chunk it is in.  (20-fold radii: merges at upload and
    on the way, in systems of one chunk and of several.)"""
    off, m, r, x, v = _systems([1, 2, 31, 64, 65, 128, 129, 256, 257, 600, 1500], inflate)
    runs = []
    for threads, bodies, cuts in ((None, None, (20,)), (64, 1, (20,)), (512, 1, (1, 19)), (256, 4, (3, 17))):
        e = Ensemble(off, m, x, v, r, dt=600.0)
        if threads:
            e.set_threads(threads)
            e.set_bodies_per_thread(bodies)
        for c in cuts:
            e.evolve(c)
        runs.append((e.counts()[:2], e.state()))
    assert (runs[0][0][1] > 0) == (inflate > 1.0)
    for counts, state in runs[1:]:
        assert np.array_equal(counts[0], runs[0][0][0]) and counts[1] == runs[0][0][1]
        for a, b in zip(state, runs[0][1]):
            for k in ("m", "r", "x", "v", "a"):
                assert np.array_equal(a[k], b[k]), k
