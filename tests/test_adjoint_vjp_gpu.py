"""The VJP kernels of the adjoint against their formula in plain torch FP64, at the positions the run itself
went through: the one-launch form at the edges of its shapes, the blocked form at the edges of tiles, row
blocks and groups, and in several batches of partial sums (from about 140000 bodies on).

With one step and the positions x0, x1 of the run, the reverse sweep from (gx, gv) is
    w = h/2 gv;  lx = gx + G J(x1)^T w;  mu = dm(x1, w);  lv = gv + h lx
    w = h/2 lv;  lx += G J(x0)^T w;      mu += dm(x0, w)
Every sum of n FP64 terms, each within a few roundings, is within (n + 16) 2^-53 of the sum of its terms'
magnitudes; the second stage takes the first one's error over, hence twice that."""
import pytest

from test_adjoint_gpu import AU, G, setup

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _vjp(x, m, w, rows):
    """(J^T w) and the mass term without G of the bodies `rows`, with the sums of their terms' magnitudes."""
    import torch
    out = [torch.empty((len(rows), 3), dtype=x.dtype, device=x.device) for _ in range(2)]
    out += [torch.empty(len(rows), dtype=x.dtype, device=x.device) for _ in range(2)]
    step = max(1, (1 << 25) // len(x))
    for b in range(0, len(rows), step):
        k = rows[b:b + step]
        d = x[None] - x[k][:, None]
        r2 = (d * d).sum(-1)
        inv3 = torch.where(r2 > 0, torch.where(r2 > 0, r2, torch.ones_like(r2)).pow(-1.5), torch.zeros_like(r2))
        wj, wk, mk = w[None], w[k][:, None], m[k][:, None]
        A, B = (wj * d).sum(-1), (wk * d).sum(-1)
        c = 3.0 * (mk * A - m[None] * B) / torch.where(r2 > 0, r2, torch.ones_like(r2))
        t = mk[..., None] * wj - m[None, :, None] * wk - c[..., None] * d
        out[0][b:b + step] = (inv3[..., None] * t).sum(1)
        # |d . w| <= |d| |w|: the magnitudes of what cancels inside a term
        big = (mk * w.norm(dim=1)[None] + m[None] * w[k].norm(dim=1)[:, None]) * inv3
        out[1][b:b + step] = (7.0 * big).sum(1)[:, None]
        out[2][b:b + step] = -(A * inv3).sum(1)
        out[3][b:b + step] = (w.norm(dim=1)[None] * r2.sqrt() * inv3).sum(1)
    return out


def _run(n, h, gx, gv):
    import torch

    from gregpackagescpp_b200.adjoint import leapfrog_final_state
    m, x, v = setup(n, n)
    leaves = [t.requires_grad_() for t in (x, v, m)]
    xT, vT = leapfrog_final_state(*leaves, G, h, 1)
    grads = torch.autograd.grad((xT, vT), leaves, (gx, gv))
    return m.detach(), x.detach(), xT.detach(), grads


@pytest.mark.parametrize("n", [2, 3, 33, 127, 592, 593, 1184, 1480, 1481, 3400, 3401, 3585, 3841, 4097, 4865])
def test_both_stages(gpu, n):
    import torch
    h = 3.0e5  # some 1e-3 of the cluster's crossing time
    gen = torch.Generator(device="cuda").manual_seed(n)
    gx, gv = (torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=gen) for _ in range(2))
    gx, gv = gx / AU, gv / 1e4
    m, x0, x1, (gx0, gv0, gm) = _run(n, h, gx, gv)
    rows = torch.arange(n, device="cuda")
    w = 0.5 * h * gv
    j1, s1, mu1, t1 = _vjp(x1, m, w, rows)
    lx = gx + G * j1
    lv = gv + h * lx
    j0, s0, mu0, t0 = _vjp(x0, m, 0.5 * h * lv, rows)
    bound = (n + 16) * U
    assert bool(((gv0 - lv).abs() <= h * bound * G * s1 + 8 * U * (gv.abs() + h * lx.abs())).all())
    assert bool(((gx0 - (lx + G * j0)).abs() <= 2 * bound * G * (s0 + s1) + 8 * U * lx.abs()).all())
    assert bool(((gm - G * (mu0 + mu1)).abs() <= 2 * bound * G * (t0 + t1)).all())


@pytest.mark.parametrize("n", [140000, 200001])
def test_batches_of_partial_sums(gpu, n):
    """From gv = 0 the second stage's w is h^2 / 2 gx exactly but for its roundings, so that a sample of
    bodies shows the sums: the first and last ones, and some of every super-group between."""
    import torch
    h = 1.0e8  # h^2 G m / r^3 of a typical pair of the cluster is not small against 1
    gen = torch.Generator(device="cuda").manual_seed(n)
    gx = torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=gen) / AU
    m, x0, _, (gx0, gv0, gm) = _run(n, h, gx, torch.zeros_like(gx))
    edges = torch.tensor([0, 1, 255, 256, 2047, 2048, n - 2049, n - 257, n - 256, n - 2, n - 1], device="cuda")
    rows = torch.cat([edges, torch.arange(77, n, 251, device="cuda")])
    assert bool((gv0 == h * gx).all())
    j0, s0, mu0, t0 = _vjp(x0, m, 0.5 * h * (h * gx), rows)
    bound = (n + 16) * U
    assert bool(((gx0[rows] - (gx[rows] + G * j0)).abs() <= bound * G * s0 + 4 * U * gx[rows].abs()).all())
    assert bool(((gm[rows] - G * mu0).abs() <= bound * G * t0).all())
    typical = ((gx0[rows] - (gx[rows] + G * j0)).abs() / (G * s0)).median()
    assert float(typical) < 64 * U  # what the sums' errors come to where none is near its bound
