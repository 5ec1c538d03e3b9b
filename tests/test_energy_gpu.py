"""System.energy at the edges of its 256-body blocks, and with the separations that add nothing."""
import numpy as np
import pytest

from gregpackagescpp_b200 import System
from gregpackagescpp_b200.ics import UNITS_G6674, plummer

pytestmark = pytest.mark.gpu
G = 6.674e-11


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 513, 3000])
def test_energy_at_block_edges(gpu, n):
    """Kinetic and potential energy against extended-precision sums; every term has one sign, so rounding
    stays at a few 2^-53 per addition chain (the 1e-13 of the oracle comparison)."""
    m, x, v = plummer(n, 7 * n)
    m = m * np.random.default_rng(n).uniform(0.0, 2.0, n)
    v = v + 1e3
    if n > 3:
        x[n // 3] = x[n - 1]  # coincident: no pair
    xl, ml = x.astype(np.longdouble), m.astype(np.longdouble)
    pe = np.longdouble(0)
    for i in range(n):
        r2 = ((xl[i + 1:] - xl[i]) ** 2).sum(1)
        ok = r2 > 0
        pe -= np.longdouble(G) * ml[i] * (ml[i + 1:][ok] / np.sqrt(r2[ok])).sum()
    ke = (0.5 * ml * (v.astype(np.longdouble) ** 2).sum(1)).sum()
    got = System(m, x, v, units_format=UNITS_G6674).energy()
    assert abs(got[0] - ke) <= 1e-13 * ke and abs(got[1] - pe) <= 1e-13 * abs(pe), (got, ke, pe)
    p = (ml[:, None] * v).sum(0)
    assert np.abs(got[2] - p).max() <= 1e-13 * np.abs(ml[:, None] * v).sum(0).max()


def test_energy_with_unusable_separations(gpu):
    """A body at infinity adds nothing; one at a subnormal squared distance adds its finite term."""
    x = np.array([[0.0, 0.0, 0.0], [np.inf, 0.0, 0.0], [3e-160, 0.0, 0.0], [1.0, 0.0, 0.0]])
    m = np.ones(4)
    _, pe, _, _ = System(m, x, np.zeros_like(x), units_format=UNITS_G6674).energy()
    assert abs(pe / (-G * (1 / np.sqrt(np.float64(3e-160) ** 2) + 2.0)) - 1) < 1e-2  # r^2 holds 4 bits there
