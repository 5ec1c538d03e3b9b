"""The adjoint's single-launch and blocked forms at their boundary, its kept and recomputed positions,
and its two kinds of memory, against torch autograd and each other."""
import pytest

from test_adjoint_gpu import AU, DT, G, setup, torch_kdk

pytestmark = pytest.mark.gpu


def _grads(n, steps, every):
    import torch

    from gregpackagescpp_b200.adjoint import leapfrog_final_state
    m, x, v = (t.requires_grad_() for t in setup(n, n))
    gen = torch.Generator(device="cuda").manual_seed(n)
    gx = torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=gen) / AU
    gv = torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=gen) / 1e4
    out = leapfrog_final_state(x, v, m, G, DT, steps, every) if every != "torch" else torch_kdk(x, v, m, steps)
    return [t.detach() for t in out] + list(torch.autograd.grad(out, (x, v, m), (gx, gv)))


@pytest.mark.parametrize("n", [2, 3, 257, 1000, 1001, 1481, 3400, 3401, 3585])
def test_forms_vs_torch(gpu, n):
    """FP64 sums of at most n terms in other orders: 1e-9 of the largest component, the bound of the
    autograd comparison, is far above their rounding."""
    got, want = _grads(n, 3, None), _grads(n, 3, "torch")
    for a, b in zip(got, want):
        assert float((a - b).abs().max() / b.abs().max()) < 1e-9


@pytest.mark.parametrize("n", [100, 3585, 4097])
def test_kept_positions_equal_recomputed_ones(gpu, n):
    kept = _grads(n, 7, None)
    for every in (1, 3, 7, 100):
        for a, b in zip(_grads(n, 7, every), kept):
            assert bool((a == b).all())


def test_own_memory_and_workspace_checks(gpu):
    import ctypes as C

    import torch

    from gregpackagescpp_b200 import _lib
    from gregpackagescpp_b200.adjoint import AdjointRun
    n, steps = 300, 4
    m, x, v = setup(n, 1)
    stream = torch.cuda.current_stream().cuda_stream
    finals = []
    for allocate in (None, lambda size: torch.empty(size, dtype=torch.uint8, device="cuda")):
        run = AdjointRun(n, steps, 2, G, DT, 0, allocate)
        xT = torch.empty_like(x)
        _lib.check(run._L.gtd_adjoint_forward(run._h, x.data_ptr(), v.data_ptr(), m.data_ptr(), xT.data_ptr(), None, stream))
        torch.cuda.synchronize()
        finals.append(xT)
    assert torch.equal(*finals)
    small = torch.empty(4096, dtype=torch.uint8, device="cuda")
    L, h = run._L, C.c_void_p()
    assert L.gtd_adjoint_create_in(C.byref(h), 0, n, steps, 2, G, DT, small.data_ptr(), 4096) == _lib.ERR_CAPACITY
    assert L.gtd_adjoint_create_in(C.byref(h), 0, n, steps, 2, G, DT, None, 1 << 30) == _lib.ERR_INVALID_ARGUMENT
