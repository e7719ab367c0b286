"""Work memory that dense string sets add (the doubles regrouped by distinct ket, csrc/sigma_union.cuh): given
back on release, and given up for a call's own vectors where memory is short."""
import pytest

from conftest import launched_kernels
from test_ab_rows import _dense

pytestmark = pytest.mark.gpu


def _problem(count):
    import synth
    from sbd_tpb import Problem
    h1, eri, core = synth.synthetic_hamiltonian(18)
    s = _dense(18, 7, count, 1)
    return Problem(norb=18, nelec=14, core=core, h1=h1, eri_packed=eri, astr=s, bstr=s.copy())


def _vector(prob):
    import torch
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.randn(prob.ndet, dtype=torch.float64, device="cuda", generator=g)
    return x, torch.empty_like(x)


def test_release_work_gives_the_lists_back():
    import torch

    import sbd_tpb
    prob = _problem(2101)
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    x, y = _vector(prob)
    h.sigma_device(x, y)
    again = launched_kernels(lambda: h.sigma_device(x, y))
    assert any("sigma_union_kernel" in k for k in again) and not any("union_fill" in k for k in again)
    ref = y.clone()
    h.free_vectors()
    assert any("union_fill" in k for k in launched_kernels(lambda: h.sigma_device(x, y)))
    assert torch.equal(y, ref)
    h.close()


def test_lists_yield_to_vectors():
    """4,041 strings: a vector is 131 MB and the lists are 52 MB.  With room for one vector and 100 MB more,
    the second vector of sbd_tpb_sigma takes the lists' place."""
    import torch

    import sbd_tpb
    prob = _problem(4041)
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    x, y = _vector(prob)
    h.sigma_device(x, y)  # C^T and the lists are there
    assert any("sigma_union_kernel" in k for k in launched_kernels(lambda: h.sigma_device(x, y)))
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    room = 8 * prob.ndet + (100 << 20)
    hold = torch.empty(free - room, dtype=torch.uint8, device="cuda")
    try:
        h.sigma(x, y)
        torch.cuda.synchronize()
    finally:
        del hold
        torch.cuda.empty_cache()
    z = h.sigma(x)  # with room again
    # another kernel for the doubles, the same terms: the same bits
    assert torch.equal(y, z)
    h.close()
