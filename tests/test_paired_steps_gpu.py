"""The callback loop's two-kernel steps (collide.cu) against the same loop run eagerly, with a kernel
each for kick-drift, force, detection and resolution: the same bits, at the edges of the sizes that
take them and just above, with and without the functors, over full, part and odd chunks of steps."""

import numpy as np
import pytest

from gregpackagescpp_b200 import RestFromCom, System, WhileRestBelow, _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 129, 900, 901, 4095, 4096, 5000])
@pytest.mark.parametrize("steps,functors", [(1, True), (64, True), (65, False), (131, True)])
def test_paired_steps_bit_identical(gpu, n, steps, functors):
    rng = np.random.default_rng(n + steps)
    edge = n ** (1.0 / 3.0)
    x = rng.uniform(-edge, edge, (n, 3))
    x[1] = x[0] + 0.1  # an overlap at any size
    v = -0.2 * x
    m, r = rng.uniform(0.5, 1.5, n), rng.uniform(0.2, 0.6, n)
    out = []
    for eager in (0, 1):
        s = System(m, x, v, r=r, rest=np.full(n, 0.7), timestep=0.05, num_iterations=steps,
                   units_format="M1:1,D1:1,T1:1", collisions=3)
        s._push()
        _lib.check(s._L.gtd_system_time_force_kernels(s._h, eager))
        fab = RestFromCom(0.5, 1.0, 4.0, 2.0, x.mean(0))
        if functors:  # never below 0: the probing count alone ends the loop
            s.evolve(System.leapfrog_kdk, WhileRestBelow(0.0, steps), None, fab)
        else:
            s.evolve(System.leapfrog_kdk, WhileRestBelow(2.0, 5), max_steps=steps)
        assert s.callback_stats()["graph_loop"] == (not eager)
        assert s.steps_taken == steps
        out.append([np.array(a) for a in (s.x, s.v, s.rest, fab.com)])
    assert np.any(out[0][1] != v)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
