"""The list walk of double trees against the per-lane walk: the same interactions, sums in another order."""
import numpy as np
import pytest

from gregpackagescpp_b200 import System
from gregpackagescpp_b200.ics import UNITS_G6674, plummer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 129, 3001])
@pytest.mark.parametrize("eps", [0.0, 1e9])
def test_double_list_walk(gpu, n, eps):
    """Equal counts; accelerations of at most n FP64 terms: 1e-12 of the largest holds their rounding.  The
    last two bodies share a full-depth code (a bucket leaf)."""
    m, x, v = plummer(n, n)
    m = m * np.random.default_rng(n).uniform(0.1, 2.0, n)
    if n > 2:
        x[n - 1] = x[n - 2] * (1 + 1e-12)
    out = []
    for variant in (1, 2):
        s = System(m, x, v, units_format=UNITS_G6674)
        s.set_bh_walk_variant(variant)
        s.set_bh_opening_angle(0.6)
        if eps:
            s.set_softening(eps)
        out.append(s.bh_accelerations(tree_float=False))
    assert np.array_equal(out[0][1], out[1][1])
    assert np.abs(out[0][0] - out[1][0]).max() <= 1e-12 * np.abs(out[0][0]).max()
