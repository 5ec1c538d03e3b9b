"""The unordered-pair kernels' queue counters are restored by each evaluation: a handle that changes its
variant, is tuned and evaluates again has the bits of one that only ever ran that variant."""
import numpy as np
import pytest

from gregpackagescpp_b200 import System, _lib
from gregpackagescpp_b200.ics import UNITS_G6674, plummer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,variants", [("f64", (5, 1, 6, 5)), ("mixed", (10, 8, 9, 10))])
@pytest.mark.parametrize("n", [4801, 9000])
def test_variants_in_turn(gpu, n, precision, variants):
    m, x, v = plummer(n, n)

    def system():
        return System(m, x, v, timestep=3600.0, num_iterations=20, units_format=UNITS_G6674, precision=precision)

    s = system()
    for k, variant in enumerate(variants):
        a = system()
        a.x, a.v = s.x, s.v
        if k == 2 and n == 9000:
            s._push()
            _lib.check(s._L.gtd_system_autotune_direct(s._h, 1, None, None))
        for h in (s, a):
            h._push()
            _lib.check(h._L.gtd_system_set_direct_variant(h._h, variant))
            h.evolve(System.leapfrog_kdk)
        assert np.array_equal(s.x, a.x) and np.array_equal(s.v, a.v), (k, variant)
        a.close()
