"""Handles without a pinned variant run one fused FP64 launch per force up to 4736 bodies, in either
precision; pinned ones above 4096 bodies, and mixed ones, run the variant."""
import os
import subprocess
import sys

import numpy as np
import pytest

from gregpackagescpp_b200 import System, _lib
from gregpackagescpp_b200.ics import UNITS_G6674, plummer

pytestmark = pytest.mark.gpu


def _system(n, precision, steps):
    m, x, v = plummer(n, n)
    return System(m, x, v, timestep=3600.0, num_iterations=steps, units_format=UNITS_G6674, precision=precision)


def _pin(s, variant):
    s._push()
    _lib.check(s._L.gtd_system_set_direct_variant(s._h, variant))


@pytest.mark.parametrize("precision,variant", [("f64", 1), ("mixed", 10)])
@pytest.mark.parametrize("n", [2, 150, 4096, 4097, 4735, 4736, 4737])
def test_fused_against_pinned(gpu, n, precision, variant):
    """The force of a free handle against a pinned one's: n rounded FP64 additions hold 1e-12 of the largest
    force many times over, mixed pair terms 1e-5 of it."""
    s = _system(n, precision, 1)
    free = s.accelerations().copy()
    _pin(s, variant)
    pinned = s.accelerations().copy()
    scale = np.abs(pinned).max()
    assert np.abs(free - pinned).max() < (1e-12 if precision == "f64" else 1e-5) * scale


@pytest.mark.parametrize("precision,variant", [("f64", 1), ("mixed", 10)])
def test_pin_between_evolves(gpu, precision, variant):
    """The steps replayed from a graph follow the handle: free, pinned and free again, each part has the
    bits of a handle that only ever ran that way."""
    n, steps = 4200, 40
    s = _system(n, precision, steps)
    s.evolve(System.leapfrog_kdk)
    a = _system(n, precision, steps)
    for pin in (variant, -1):
        a.x, a.v = s.x, s.v
        _pin(s, pin)
        _pin(a, pin)
        s.evolve(System.leapfrog_kdk)
        a.evolve(System.leapfrog_kdk)
        assert np.array_equal(s.x, a.x) and np.array_equal(s.v, a.v)
        a.close()
        a = _system(n, precision, steps)


def test_mixed_runs_fp64_kernel(gpu):
    """A free mixed handle has the FP64 handle's bits up to 4736 bodies and not above.  In a process of its
    own: a handle is free only where nobody in the process has tuned its size."""
    code = ("import sys; sys.path.insert(0, 'tests'); import numpy as np; from test_fused_auto_gpu import _system\n"
            "print([np.array_equal(*(_system(n, p, 1).accelerations() for p in ('f64', 'mixed')))"
            " for n in (2, 150, 4096, 4097, 4736, 4737)])")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=root, timeout=300)
    assert out.stdout.strip() == "[True, True, True, True, True, False]", out.stdout + out.stderr
