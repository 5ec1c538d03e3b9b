"""A handle whose bodies do not fit the device holds none: it can be stepped, read and uploaded again."""
import numpy as np
import pytest

from gregpackagescpp_b200 import System, _lib
from gregpackagescpp_b200.ics import UNITS_G6674, plummer

pytestmark = pytest.mark.gpu


def test_more_bodies_than_memory(gpu):
    """2^31 - 1 bodies take 64 GiB an array of four doubles; the arrays are not read before they fit."""
    import ctypes as C
    m, x, v = plummer(500, 1)
    s = System(m, x, v, timestep=3600.0, num_iterations=3, units_format=UNITS_G6674)
    s.evolve(System.leapfrog_kdk)
    want = s.x.copy()
    L, n, ns = s._L, C.c_int64(1), C.c_int64()
    rc = L.gtd_system_upload(s._h, 2 ** 31 - 1, _lib.ptr(m), None, None, _lib.ptr(x), None)
    assert rc == _lib.ERR_OUT_OF_MEMORY
    assert L.gtd_system_num_bodies(s._h, C.byref(n)) == 0 and n.value == 0
    assert L.gtd_system_evolve(s._h, System.leapfrog_kdk, C.byref(ns)) == 0
    s.m, s.x, s.v = m, x, v
    s.evolve(System.leapfrog_kdk)
    assert np.array_equal(s.x, want)
