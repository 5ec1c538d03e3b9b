"""The ensemble's smallest systems: a warp of the force loop has more lanes than the system rows."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from gregpackagescpp_b200.ensemble import Ensemble
from gregpackagescpp_b200.ics import AU, ensemble

HERE = os.path.dirname(os.path.abspath(__file__))


def test_reads_stay_in_the_staged_rows(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "ens_rows"
    subprocess.run([nvcc, "-O1", "-std=c++17", "-I" + os.path.join(os.path.dirname(HERE), "gregpackagescpp_b200", "csrc"),
                    os.path.join(HERE, "cpp", "ens_rows_main.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("bodies", [1, 2, 4])
@pytest.mark.parametrize("n", [1, 2, 3, 14, 31, 33])
def test_smallest_systems(gpu, oracle, n, bodies):
    """Two systems of n bodies, the largest of their ensemble, for 20 steps against the oracle's FP64 run.
    FP32 pair terms (6e-8 of a force each) over 20 steps of 600 s move a body by less than 1e-6 of the
    path that its acceleration alone covers; the starting state dominates x and v, 1e-9 and 1e-7 of it."""
    parts = [ensemble(1, 400 + n + k, n_min=n, n_max=n, r_ball=2.0 * AU)[1:] for k in range(2)]
    m, r, x, v = (np.concatenate(a) for a in zip(*parts))
    e = Ensemble(np.array([0, n, 2 * n]), m, x, v, r, merge=False, dt=600.0)
    e.set_threads(128)
    e.set_bodies_per_thread(bodies)
    e.evolve(20)
    for k, st in enumerate(e.state()):
        s = slice(k * n, (k + 1) * n)
        xo, vo, _ = oracle.evolve(16, m[s], x[s], v[s], 600.0, 20, oracle.G("M66743:66740,D1:1,T1:1"))
        assert np.abs(st["x"] - xo).max() <= 1e-9 * np.abs(xo).max()
        assert np.abs(st["v"] - vo).max() <= 1e-7 * np.abs(vo).max()
