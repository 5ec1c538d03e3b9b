"""Copies between pageable arrays and the device by several threads (csrc/host_copy.cu), over a stand-in for
the CUDA runtime: partial last chunks, arrays that are pinned already, several handles, memory that cannot
be pinned and an error in the middle."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_ring_copies(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.fail("no CUDA headers at " + include)
    exe = tmp_path / "host_copy"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I" + include, "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "gregpackagescpp_b200", "csrc"), os.path.join(HERE, "cpp", "host_copy_main.cpp"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout


@pytest.mark.gpu
def test_arrays_there_and_back(gpu):
    """A handle's arrays come back as they went in, before, at and after the copies that make its ring."""
    from gregpackagescpp_b200 import System
    rng = np.random.default_rng(5)
    n = 200003
    s = System(np.ones(n), np.zeros((n, 3)), np.zeros((n, 3)))
    for k in range(5):
        s.m, s.r, s.rest = rng.uniform(0, 1, n), rng.uniform(0, 1, n), rng.uniform(0, 1, n)
        s.x, s.v = rng.normal(size=(n, 3)), rng.normal(size=(n, 3))
        want = [a.copy() for a in (s.m, s.r, s.rest, s.x, s.v)]
        s._push()
        s.m, s.r, s.rest, s.x, s.v = (np.zeros_like(a) for a in want)
        s._pull()
        for a, b in zip((s.m, s.r, s.rest, s.x, s.v), want):
            assert np.array_equal(a, b), k
