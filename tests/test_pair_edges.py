"""Small direct sums against host sums in FP64: every launch shape of the fused kernel at its edges, in
either precision, as a force of a handle, of the no-allocation entry and of a step; and the index
arithmetic of the adjoint's unordered pairs on the host."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from gregpackagescpp_b200 import System, _lib
from gregpackagescpp_b200.ics import UNITS_G6674, plummer
from test_direct_sym import G, _host_acc

HERE = os.path.dirname(os.path.abspath(__file__))
# {1, 2, 4} up to 128 and 592 bodies, {2, 1, 5} 1480, {2, 1, 8} 2368, {4, 2, 3} 3552, {2, 1, 8} above; chunks of
# 128 bodies a round, one to four rounds in flight
EDGES = [1, 31, 127, 128, 129, 255, 256, 257, 385, 512, 513, 592, 593, 641, 1480, 1481, 2368, 2369, 3552, 3553, 4096]


def test_vjp_units_and_slots(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "sym_units_vjp"
    csrc = os.path.join(os.path.dirname(HERE), "gregpackagescpp_b200", "csrc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O1", "-std=c++17", "-I" + csrc,
                    "-I" + os.path.join(os.path.dirname(HERE), "include"), os.path.join(HERE, "cpp", "sym_units_vjp_main.cu"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout


def _bodies(n):
    m, x, v = plummer(n, n + 7)
    m = m * np.random.default_rng(n).uniform(0.0, 2.0, n)
    m[::5] = 0.0
    if n > 2:
        x[n - 1] = x[0]  # coincident: no pair
    return m, x, v


def _close(got, want, scale, n):
    """n FP64 terms, each within a few roundings of its own: (n + 16) 2^-53 of the terms' magnitudes."""
    return (np.abs(got - want) <= 2 * (n + 16) * 2.0 ** -53 * scale[:, None] + 1e-300).all()


@pytest.mark.gpu
@pytest.mark.parametrize("n", EDGES + [4097, 4735, 4736])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_forces(gpu, n, precision):
    import torch
    m, x, v = _bodies(n)
    want, scale = _host_acc(m, x)
    s = System(m, x, v, units_format=UNITS_G6674, precision=precision)
    assert _close(s.accelerations(), want, scale, n)
    pm4 = torch.tensor(np.concatenate([x, m[:, None]], 1), device="cuda")
    acc = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
    fn = _lib.load().gtd_direct_accelerations_noalloc
    fn.argtypes = [C.c_int64, C.c_void_p, C.c_double, C.c_int, C.c_void_p, C.c_void_p]
    _lib.check(fn(n, pm4.data_ptr(), G, _lib.PREC_F64 if precision == "f64" else _lib.PREC_MIXED, acc.data_ptr(),
                  torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert _close(acc.cpu().numpy(), want, scale, n)


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["leapfrog_kdk", "leapfrog_dkd", "euler", "modified_euler", "midpoint"])
@pytest.mark.parametrize("n", [128, 129, 592, 593])
def test_steps(gpu, n, method):
    """Two steps from host sums; 1e-12 of the largest position and velocity as in the other step tests."""
    m, x, v = _bodies(n)
    h = 3600.0
    s = System(m, x, v, timestep=h, num_iterations=2, units_format=UNITS_G6674)
    s.evolve(getattr(System, method))

    def acc(p):
        return _host_acc(m, p)[0]

    for _ in range(2):
        if method == "leapfrog_kdk":
            v = v + 0.5 * h * acc(x)
            x = x + h * v
            v = v + 0.5 * h * acc(x)
        elif method == "leapfrog_dkd":
            x = x + 0.5 * h * v
            v = v + h * acc(x)
            x = x + 0.5 * h * v
        elif method == "euler":
            x, v = x + h * v, v + h * acc(x)
        elif method == "modified_euler":
            a = acc(x)
            vp = v + h * a
            ap = acc(x + h * v)
            x, v = x + 0.5 * h * (v + vp), v + 0.5 * h * (a + ap)
        else:
            a = acc(x)
            vp = v + 0.5 * h * a
            ap = acc(x + 0.5 * h * v)
            x, v = x + h * vp, v + h * ap
    assert np.abs(s.x - x).max() <= 1e-12 * np.abs(x).max()
    assert np.abs(s.v - v).max() <= 1e-12 * np.abs(v).max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1184, 1185])
def test_paired_blocks(gpu, n):
    """The callback loop's two-kernel steps where a block starts to hold two bodies."""
    import test_paired_steps_gpu as paired
    paired.test_paired_steps_bit_identical(gpu, n, 65, True)
