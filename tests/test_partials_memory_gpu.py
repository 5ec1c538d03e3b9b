"""A handle whose partial sums do not fit the memory that is left evaluates its force in smaller batches."""
import numpy as np
import pytest

from gregpackagescpp_b200 import System
from gregpackagescpp_b200.ics import UNITS_G6674, plummer

pytestmark = pytest.mark.gpu


def _fill(leave):
    """Takes the device's free memory but about `leave` bytes."""
    import torch
    held, size = [], 16 << 30
    while size >= 4 << 20:
        if torch.cuda.mem_get_info()[0] < leave + size:
            size >>= 1
            continue
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size >>= 1
    return held


@pytest.mark.parametrize("leave", [128 << 20, 32 << 20])
def test_force_and_steps_with_little_memory(gpu, leave):
    """65536 bodies take 201 MB of partial sums in one batch.  In smaller ones each body's sum takes its terms
    in another order: 1e-12 of the largest force is n rounded FP64 additions many times over."""
    import torch
    n = 65536
    m, x, v = plummer(n, 3)

    def system():
        return System(m, x, v, timestep=3600.0, num_iterations=18, units_format=UNITS_G6674)

    s = system()
    want = s.accelerations().copy()
    s.evolve(System.leapfrog_kdk)
    xw = s.x.copy()
    s.close()
    s = system()
    s._push()
    held = _fill(leave)
    try:
        assert torch.cuda.mem_get_info()[0] < leave + (16 << 20)
        got = s.accelerations().copy()
        s.evolve(System.leapfrog_kdk)  # steps replayed from a graph as well
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
    assert np.abs(s.x - xw).max() <= 1e-12 * np.abs(xw).max()
    assert np.array_equal(s.accelerations(), s.accelerations())
