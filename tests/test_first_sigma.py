"""What the first sigma of a new problem does beside the later ones: copies of tables to the host,
allocations and kernels that set it up."""
import numpy as np
import pytest

from conftest import traced

pytestmark = pytest.mark.gpu


def _first(norb, ne, count):
    """Runtime calls and GPU activities of the first sigma of a handle, another one being there already
    (memory that the driver keeps and code that it loads once are not the handle's)."""
    import torch

    import sbd_tpb
    import synth
    h1, eri, core = synth.synthetic_hamiltonian(norb)
    s = synth.sample_strings(norb, ne, count)
    prob = sbd_tpb.Problem(norb=norb, nelec=2 * ne, core=core, h1=h1, eri_packed=eri, astr=s, bstr=s.copy())
    x = torch.from_numpy(np.random.default_rng(1).normal(size=prob.ndet)).cuda()
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    hs = [sbd_tpb.Handle(0) for _ in range(2)]
    for h in hs:
        h.set_problem(prob)
        got = traced(lambda: h.sigma_device(x, y))
    for h in hs:
        h.close()
    return got


def test_set_up_of_a_small_problem():
    """8-orbital full CI: the row program is one allocation, and no memory is pinned for it (a pinned word per
    handle took the first sigma from 0.5 to 3 ms, the time of 40 sigmas)."""
    calls, gpu = _first(8, 4, 70)
    assert any("ab_rows_kernel" in k for k in gpu)  # the trace sees the path
    assert not [c for c in calls if c in ("cudaHostAlloc", "cudaMallocHost")]
    # the row program, C^T, and per spin the Coulomb table, its pairs' map and the list it is made from
    assert len([c for c in calls if c == "cudaMalloc"]) <= 8, calls


def test_set_up_where_the_dense_paths_do_not_run():
    """A sampled set takes the per-row passes and the direct alpha-beta kernel: asking whether it should
    copies each table once and launches nothing."""
    calls, gpu = _first(24, 8, 1500)
    assert any("ab_sparse_kernel" in k for k in gpu)
    assert not [k for k in gpu if "union" in k or "ab_rows" in k]
    # offsets of both spins, kets and pairs of the beta singles; pairs of each spin for the Coulomb tables
    assert len([k for k in gpu if "DtoH" in k]) <= 6, gpu
