"""An ensemble whose upload was refused holds no systems: it can be stepped, read and uploaded again."""
import ctypes as C

import numpy as np
import pytest

from gregpackagescpp_b200 import _lib
from gregpackagescpp_b200.ensemble import Ensemble
from gregpackagescpp_b200.ics import ensemble

pytestmark = pytest.mark.gpu


def test_refused_and_empty_uploads(gpu):
    off, m, r, x, v = ensemble(3, 5, n_min=40, n_max=60)
    e = Ensemble(off, m, x, v, r, dt=60.0)
    e.evolve(3)
    want = e.state()
    L, ptr = e._L, _lib.ptr

    def upload(offsets, mass):
        return L.gtd_ensemble_upload(e._h, len(offsets) - 1, ptr(offsets), ptr(mass), ptr(r), None, ptr(x), ptr(v))

    def holds_nothing():
        ns, merges = C.c_int64(1), C.c_uint64(1)
        assert L.gtd_ensemble_evolve(e._h, 5, C.byref(ns)) == 0 and ns.value == 0
        assert L.gtd_ensemble_counts(e._h, None, C.byref(merges), None) == 0 and merges.value == 0
        assert L.gtd_ensemble_download(e._h, None, None, None, None, None, None) == 0

    negative = m.copy()
    negative[7] = -1.0
    for offsets, mass, rc in ((off[::-1].copy(), m, _lib.ERR_INVALID_ARGUMENT), (off, negative, _lib.ERR_INVALID_ARGUMENT),
                              (np.array([0, 9000], dtype=np.int64), np.ones(9000), _lib.ERR_CAPACITY)):
        assert upload(offsets, mass) == rc
        holds_nothing()
    assert L.gtd_ensemble_upload(e._h, 0, None, None, None, None, None, None) == 0
    holds_nothing()
    assert upload(off, m) == 0
    e.evolve(3)
    for a, b in zip(e.state(), want):
        assert all(np.array_equal(a[k], b[k]) for k in ("m", "r", "x", "v"))
