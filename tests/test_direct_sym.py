"""The direct-sum kernels that evaluate each unordered pair once (csrc/direct_sym.cu): their index
arithmetic on the host, and their forces on the GPU at the edges of tiles, row blocks and groups."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from gregpackagescpp_b200 import System, _lib
from gregpackagescpp_b200.ics import UNITS_G6674, plummer

HERE = os.path.dirname(os.path.abspath(__file__))
G = 6.674e-11


def test_units_cover_every_pair_once(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "sym_units"
    subprocess.run([nvcc, "-O1", "-std=c++17", "-I" + os.path.join(os.path.dirname(HERE), "gregpackagescpp_b200", "csrc"),
                    os.path.join(HERE, "cpp", "sym_units_main.cu"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout


def _host_acc(m, x):
    """Accelerations and force scales sum_j G m_j / r^2 in FP64; a pair at zero distance adds nothing."""
    a, scale = np.empty_like(x), np.empty(len(m))
    for b in range(0, len(m), 256):
        d = x[None] - x[b:b + 256, None]
        r2 = (d * d).sum(2)
        w = np.where(r2 > 0, G * m / np.where(r2 > 0, r2, 1.0), 0.0)
        scale[b:b + 256] = w.sum(1)
        a[b:b + 256] = ((w / np.sqrt(np.where(r2 > 0, r2, 1.0)))[:, :, None] * d).sum(1)
    return a, scale


@pytest.mark.gpu
@pytest.mark.parametrize("precision,n", [("f64", n) for n in (4097, 4608, 4609, 5121, 8193)] +
                         [("mixed", n) for n in (2, 33, 64, 65, 128, 513, 1024, 1025, 2561, 4097)])
def test_forces_at_block_edges(gpu, n, precision):
    """Unequal masses, massless bodies, a distant body, and two coincident ones in one group.  FP64 (handles
    of more than 4096 bodies; smaller ones run the fused kernel): n rounded additions per component, 1e-12
    of the force scale holds that many times over; mixed: the documented 1e-6 of the force scale."""
    m, x, _ = plummer(n, n)
    m = m * np.random.default_rng(n).uniform(0.0, 2.0, n)
    m[::7] = 0.0
    x[n // 2] *= 40.0
    if n > 64:
        x[40] = x[41]
    want, scale = _host_acc(m, x)
    scale = np.maximum(scale, 1e-300)
    for variant in (5, 6) if precision == "f64" else (9, 10):
        s = System(m, x, np.zeros_like(x), units_format=UNITS_G6674, precision=precision)
        _lib.check(s._L.gtd_system_set_direct_variant(s._h, variant))
        err = np.linalg.norm(s.accelerations() - want, axis=1) / scale
        assert err.max() < (1e-12 if precision == "f64" else 1e-6), (variant, err.max(), int(err.argmax()))


@pytest.mark.gpu
@pytest.mark.parametrize("n,precision", [(300, "f64"), (4096, "f64"), (4097, "f64"), (12289, "f64"), (60001, "f64"),
                                         (7, "mixed"), (1000, "mixed"), (65536, "mixed")])
def test_noalloc_paths(gpu, n, precision):
    """gtd_direct_accelerations_noalloc through its fused, single-batch and batched forms against the
    ordered-pair kernels of a handle."""
    import torch
    m, x, v = plummer(n, 5)
    pm4 = torch.tensor(np.concatenate([x, m[:, None]], 1), device="cuda")
    acc = torch.full((n, 3), float("nan"), dtype=torch.float64, device="cuda")
    fn = _lib.load().gtd_direct_accelerations_noalloc
    fn.argtypes = [C.c_int64, C.c_void_p, C.c_double, C.c_int, C.c_void_p, C.c_void_p]
    _lib.check(fn(n, pm4.data_ptr(), G, _lib.PREC_F64 if precision == "f64" else _lib.PREC_MIXED, acc.data_ptr(),
                  torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    s = System(m, x, v, units_format=UNITS_G6674)
    _lib.check(s._L.gtd_system_set_direct_variant(s._h, 2))
    want = s.accelerations()
    rel = np.linalg.norm(acc.cpu().numpy() - want, axis=1) / np.linalg.norm(want, axis=1)
    if precision == "f64":
        assert rel.max() < 1e-12, rel.max()
    else:
        assert np.sqrt((rel ** 2).mean()) < 1e-6, rel.max()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 3, 900, 901, 1480, 1481, 2368, 2369, 3551, 3552, 3553, 4095])
def test_fused_shapes(gpu, n):
    """Every launch shape of the fused FP64 kernel at its boundary, odd counts included, under a two-stage
    method: the positions and velocities of one modified Euler step from host sums (FP64, 1e-12)."""
    m, x, v = plummer(n, n)
    x[n - 1] = x[0]  # coincident: no pair
    h = 3600.0
    a, _ = _host_acc(m, x)
    xp, vp = x + h * v, v + h * a
    ap, _ = _host_acc(m, xp)
    s = System(m, x, v, timestep=h, num_iterations=1, units_format=UNITS_G6674)
    s.evolve(System.modified_euler)
    for got, want in ((s.x, x + 0.5 * h * (v + vp)), (s.v, v + 0.5 * h * (a + ap)), (s.a, a)):
        assert np.abs(got - want).max() <= 1e-12 * np.abs(want).max()
