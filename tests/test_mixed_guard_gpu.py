"""Coincident bodies under the mixed pair kernels' unguarded fast path: where the close-pair check is off,
and where a whole warp's rows lie at the centre of their frame, they are selected away within the aligned
runs of 1024 bodies (as in the FP64 kernel for these sizes and the ordered mixed one)."""
import numpy as np
import pytest

from gregpackagescpp_b200 import System, _lib
from gregpackagescpp_b200.ics import UNITS_G6674, plummer

pytestmark = pytest.mark.gpu


def _accelerations(m, x, precision, variant=-1, near=None):
    # overlap collisions keep the bodies in the order given
    s = System(m, x, np.zeros_like(x), r=np.zeros(len(m)), units_format=UNITS_G6674, precision=precision, collisions=3)
    s._push()
    _lib.check(s._L.gtd_system_set_direct_variant(s._h, variant))
    if near is not None:
        _lib.check(s._L.gtd_system_set_mixed_near_factor(s._h, near))
    return s.accelerations()


def _rms(got, want):
    return np.sqrt((((got - want) ** 2).sum(1) / (want ** 2).sum(1)).mean())


@pytest.mark.parametrize("variant", [-1, 9, 10])
@pytest.mark.parametrize("i,j", [(300, 700), (511, 512), (1500, 1700), (32768 + 20, 32768 + 230)])
def test_check_off(gpu, i, j, variant):
    """Without the check a pair at distance d carries 2^-24 R / d of its term, R the cluster: 1e-4 of a body's
    acceleration, root mean square, is more than that for the nearest neighbours of 33000 bodies (R / 30)."""
    m, x, _ = plummer(33000, 17)
    x[j] = x[i]
    got = _accelerations(m, x, "mixed", variant, 1.0)
    assert np.isfinite(got).all()
    assert _rms(got, _accelerations(m, x, "f64")) < 1e-4


def test_rows_at_the_centre(gpu):
    """1024 bodies at the origin, the documented 1e-6 with the check as it is by default."""
    m, x, _ = plummer(33000, 18)
    x[2048:3072] = 0.0
    got = _accelerations(m, x, "mixed")
    assert np.isfinite(got).all()
    assert _rms(got, _accelerations(m, x, "f64")) < 1e-6
