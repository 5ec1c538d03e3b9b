"""gtd_system_autotune_direct never leaves a handle on a slower kernel: at the sizes of the fused FP64
launch, which no variant beats, tuning changes nothing for a handle without a pinned variant."""
import ctypes as C

import numpy as np
import pytest

from gregpackagescpp_b200 import System, _lib
from gregpackagescpp_b200.ics import UNITS_G6674, plummer

pytestmark = pytest.mark.gpu


def _system(n, precision):
    m, x, v = plummer(n, n)
    s = System(m, x, v, timestep=3600.0, num_iterations=20, units_format=UNITS_G6674, precision=precision)
    s._push()
    return s


def _tune(s, reps=1):
    best = C.c_int()
    _lib.check(s._L.gtd_system_autotune_direct(s._h, reps, C.byref(best), None))
    return best.value


@pytest.mark.parametrize("tuned", ["itself", "another"])
@pytest.mark.parametrize("n,precision", [(100, "mixed"), (1024, "mixed"), (4700, "mixed"), (1024, "f64"), (4700, "f64")])
def test_tuning_keeps_the_fused_launch(gpu, n, precision, tuned):
    """Tuned itself, or by another handle of its size class: force and steps have the bits and the number
    of launches of a handle nobody tuned; a pinned variant is still taken (mixed: FP32 pair terms)."""
    want = _system(n, precision)
    before = want.launch_count()
    a = want.accelerations()
    launches = want.launch_count() - before
    want.evolve(System.leapfrog_kdk)
    s, other = _system(n, precision), _system(n + (n & 1) + 1, precision)
    best = _tune(s if tuned == "itself" else other)
    before = s.launch_count()
    assert np.array_equal(s.accelerations(), a)
    assert s.launch_count() - before == launches
    s.evolve(System.leapfrog_kdk)
    assert np.array_equal(s.x, want.x) and np.array_equal(s.v, want.v)
    if precision == "mixed":
        p = _system(n, precision)
        _lib.check(p._L.gtd_system_set_direct_variant(p._h, best))
        assert not np.array_equal(p.accelerations(), a)


def test_whole_evaluations_are_timed(gpu):
    """A variant is judged by its force kernel and the sum of its partial sums: both run, reps + 1 times per
    variant (two launches each at this size), and the bodies and what a step gives from them stay."""
    n, reps = 9000, 2
    want, s = _system(n, "f64"), _system(n, "f64")
    count, before = C.c_int(), s.launch_count()
    _lib.check(s._L.gtd_direct_variant_count(_lib.PREC_F64, C.byref(count)))
    best = _tune(s, reps)
    assert s.launch_count() - before == count.value * (reps + 1) * 2
    _lib.check(want._L.gtd_system_set_direct_variant(want._h, best))
    for h in (s, want):
        h.evolve(System.leapfrog_kdk)
    assert np.array_equal(s.x, want.x) and np.array_equal(s.v, want.v)


def test_tuning_while_a_graph_is_captured(gpu):
    """Another thread tunes the size class while the callback loop is being captured (a hook runs then): the
    handle keeps the variant that the run began with, and the loop stays a graph."""
    import threading

    from gregpackagescpp_b200 import DeviceHook
    n = 6000
    small, large, s, want = (_system(k, "f64") for k in (4200, 8191, n, n))
    first = _tune(large)
    _lib.check(want._L.gtd_system_set_direct_variant(want._h, first))
    seen = []

    def tune():
        # 4200 and 8191 bodies have other fastest variants; take turns until the choice differs
        for h in (small, large, small):
            seen.append(_tune(h))
            if seen[-1] != first:
                break

    @C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p)
    def hook(user, bodies):
        if not seen:
            t = threading.Thread(target=tune)
            t.start()
            t.join()
        return 0

    each = DeviceHook(C.cast(hook, C.c_void_p).value)
    none = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p)(lambda user, bodies: 0)
    s.evolve(System.leapfrog_kdk, None, each, None)
    assert seen and seen[-1] != first, (first, seen)
    assert s.callback_stats()["graph_loop"]
    want.evolve(System.leapfrog_kdk, None, DeviceHook(C.cast(none, C.c_void_p).value), None)
    assert np.array_equal(s.x, want.x) and np.array_equal(s.v, want.v)
