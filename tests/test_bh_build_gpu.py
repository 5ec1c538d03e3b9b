"""The Barnes-Hut build at the edges of its sort (chunks of 2048 keys, groups of 16 blocks) and of its
levels of moments, bit-exact against the host rebuild, and the forces on the bodies it lays out."""
import numpy as np
import pytest

from gregpackagescpp_b200 import System
from gregpackagescpp_b200.ics import UNITS_G6674, plummer
from test_octree_gpu import compare_tree, gpu_tree

pytestmark = pytest.mark.gpu


def _check(oracle, m, x, tree_float):
    s, t = gpu_tree(m, x, tree_float)
    o = oracle.bh_tree(x, m, tree_float)
    try:
        compare_tree(t, o)
    finally:
        oracle.bh_free(o)
    return t


@pytest.mark.parametrize("tree_float", [0, 1])
@pytest.mark.parametrize("n", [2047, 2048, 2049, 32767, 32768, 32769, 34817])
def test_build_at_sort_edges(gpu, oracle, n, tree_float):
    m, x, _ = plummer(n, n)
    _check(oracle, m, x, tree_float)


@pytest.mark.parametrize("tree_float", [0, 1])
def test_build_depths(gpu, oracle, tree_float):
    """The shallowest tree with an internal level below the root's and one whose pair parts at the last."""
    m = np.ones(9)
    x = np.array([[i & 1, i >> 1 & 1, i >> 2 & 1] for i in range(8)] + [[0.9, 0.9, 0.9]], float)
    t = _check(oracle, m, x, tree_float)
    assert t["depth"].max() <= 3
    x[8] = x[7] - 2.0 ** -20
    t = _check(oracle, m, x, tree_float)
    assert t["depth"].max() >= 20


@pytest.mark.parametrize("tree_float", [0, 1])
def test_forces_on_laid_out_bodies(gpu, tree_float):
    """With theta = 0 every body meets every other as a leaf: the direct sum, to the walk's precision."""
    m, x, v = plummer(3000, 5)
    s = System(m, x, v, units_format=UNITS_G6674)
    want = s.accelerations().copy()
    s.set_bh_opening_angle(0.0)
    got = s.bh_accelerations(bool(tree_float))
    got = got[0] if isinstance(got, tuple) else got
    err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() < (1e-4 if tree_float else 1e-12)


@pytest.mark.parametrize("run", [31, 32, 33, 1000])
def test_build_with_runs_of_equal_prefixes(gpu, oracle, run):
    """A cluster whose bodies share all that the five passes of the build's sort order by, up to the length
    that is sorted in place and beyond (the full sort, which the handle's next builds take at once)."""
    rng = np.random.default_rng(run)
    x = np.concatenate([rng.uniform(0.0, 1.0, (500, 3)), 0.3 + rng.uniform(0.0, 2.0 ** -17, (run, 3))])
    x = np.ascontiguousarray(x[rng.permutation(len(x))])
    m = rng.uniform(0.5, 1.5, len(x))
    s, t = gpu_tree(m, x, 0)
    o = oracle.bh_tree(x, m, 0)
    try:
        compare_tree(t, o)
        s.bh_build(0)
        compare_tree(s.bh_tree(), o)
    finally:
        oracle.bh_free(o)
