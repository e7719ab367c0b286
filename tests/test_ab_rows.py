"""Sigma on densely connected string sets -- the alpha-beta term (csrc/ab_rows.cu: one product per alpha
row and a gather over the beta singles) and the same-spin passes (csrc/sigma_union.cuh from 8,192
determinants per SM, one row per thread below) -- against the oracle, at the sizes where their tiling can
go wrong.

Sets: n strings of lowest orbital-index sum with noise, so that they hold tens of singles each.  Column
steps are 32 wide, rows of the product come in blocks of 8 (one pass up to 24 blocks), singles in groups
of 64, and a sigma row that does not fit shared memory is summed in a scratch row.
"""
import itertools

import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


def _dense(norb, n, count, seed):
    idx = np.array(list(itertools.combinations(range(norb), n)), np.int64)
    score = idx.sum(axis=1) + 2.0 * np.random.default_rng(seed).gumbel(size=len(idx))
    score[0] = -np.inf
    keep = np.argsort(score, kind="stable")[:count]
    return np.sort((np.int64(1) << idx[keep]).sum(axis=1).astype(np.uint64))


SMS = 148

CASES = {
    # norb, (alpha electrons, strings), (beta electrons, strings): what is at its edge
    "full8": (8, (4, 70), (4, 70)),            # 28 pairs: the last block of 8 rows half empty
    "full7_33": (7, (3, 35), (2, 21)),         # fewer columns than one step
    "chunk_exact": (12, (4, 256), (4, 256)),   # whole steps, last one full
    "chunk_plus1": (12, (4, 257), (4, 257)),   # last step one column
    "two_groups": (18, (7, 600), (7, 600)),    # up to 77 singles in a row: two groups of at most 64
    "two_passes": (24, (5, 401), (4, 333)),    # up to 276 pairs: two passes over the rows of the product
    "one_row": (10, (5, 2), (5, 252)),         # rows with a single single
    "union": (18, (7, 1101), (7, 1103)),       # just above the line of the union passes: narrow FP32 tiles
    "many_blocks": (18, (7, 1400), (7, 2101)),  # the widest thread tiles of the same-spin passes, odd rows
    "union_sym": (18, (7, 1400), (7, 1400)),   # the one-pass form on the union passes (FP64)
    "two_passes_sym": (24, (5, 1301), (5, 1301)),  # 276 pairs, two passes, each with its triangle of the terms
    "wide": (18, (7, 24), (7, 15001)),         # a sigma row longer than shared memory holds in FP64
    "wide_rows": (18, (7, 301), (7, 9001)),    # the same with more rows than SMs
}


def _problem(name):
    import synth
    from sbd_tpb import Problem
    norb, (ea, na), (eb, nb) = CASES[name]
    h1, eri, core = synth.synthetic_hamiltonian(norb, seed=5)
    a = _dense(norb, ea, na, 1)
    b = a.copy() if (ea, na) == (eb, nb) else _dense(norb, eb, nb, 2)
    return Problem(norb=norb, nelec=ea + eb, core=core, h1=h1, eri_packed=eri, astr=a, bstr=b)


def _oracle_rows(prob, x, rows):
    import pyoracle
    ham = pyoracle.Hamiltonian.from_arrays(prob.norb, prob.nelec, prob.core, prob.h1, prob.eri_packed)
    return pyoracle.System(ham, prob.astr, prob.bstr).sigma_rows(rows, x)


@pytest.mark.parametrize("name", sorted(CASES))
def test_alpha_beta_rows_against_oracle(name):
    import sbd_tpb
    prob = _problem(name)
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    rng = np.random.default_rng(7)
    x = rng.normal(size=prob.ndet)
    rows = np.sort(rng.choice(prob.ndet, size=min(300, prob.ndet), replace=False)).astype(np.uint64)
    ref = _oracle_rows(prob, x, rows)
    ran = launched_kernels(lambda: h.sigma(x))
    assert any("ab_rows_kernel" in k for k in ran)
    assert any("sigma_union_kernel" in k for k in ran) == (prob.ndet >= 8192 * SMS)
    out = h.sigma(x)
    assert np.array_equal(out, h.sigma(x))  # one owner per element: the same bits again
    scale = float(np.max(np.abs(ref)))
    # FP64 sums of the same terms in another order
    assert float(np.max(np.abs(out[rows] - ref))) <= 1e-12 * scale
    # FP32: vectors and results rounded to FP32, 2^-24 a value over a few thousand terms of random sign
    out32 = h.sigma(x.astype(np.float32)).astype(np.float64)
    assert float(np.max(np.abs(out32[rows] - ref))) <= 2e-6 * scale
    h.close()


@pytest.mark.parametrize("name", [n for n in sorted(CASES) if CASES[n][1] == CASES[n][2]])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_alpha_beta_rows_symmetric_half(name, dtype):
    """The symmetric form adds only the half of the terms whose transposes are the other half."""
    import torch

    import sbd_tpb
    prob = _problem(name)
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    n = len(prob.astr)
    g = torch.Generator(device="cuda").manual_seed(3)
    r = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    x = (r + r.T).to(getattr(torch, dtype)).reshape(-1).contiguous()
    ref, out = torch.zeros_like(x), torch.full_like(x, float("nan"))
    torch.cuda.synchronize()  # the library runs on a stream of its own
    h.sigma_device(x, ref)
    ran = launched_kernels(lambda: h.sigma_device(x, out, symmetric=True))
    if dtype == "float64":
        assert any("ab_rows_kernel" in k for k in ran)
        assert any("sigma_union_kernel" in k for k in ran) == (prob.ndet >= 8192 * SMS)
    err = float((out.double() - ref.double()).abs().max()) / float(ref.double().abs().max())
    assert err <= (1e-13 if dtype == "float64" else 3e-6), err
    h.close()


def test_wide_rows_lose_no_digits():
    """A row of sums that does not fit in shared memory (FP32 above some 35,000 columns) is summed from zero
    as well: the FP32 sigma stays within the rounding of its own result (2^-24 / sqrt(3) = 3.4e-8 of its norm)
    and of sums of some hundred FP32 terms about as large.  Added to sigma one by one the terms cost 1.7e-7."""
    import torch

    import sbd_tpb
    import synth
    norb, na, nb = 20, 24, 40001
    h1, eri, core = synth.synthetic_hamiltonian(norb, seed=5)
    prob = sbd_tpb.Problem(norb=norb, nelec=14, core=core, h1=h1, eri_packed=eri, astr=_dense(norb, 7, na, 1),
                           bstr=_dense(norb, 7, nb, 1))
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn(prob.ndet, dtype=torch.float32, device="cuda", generator=g)
    y, ref = torch.zeros_like(x), torch.zeros(prob.ndet, dtype=torch.float64, device="cuda")
    h.sigma_device(x.double(), ref)
    assert any("ab_rows_kernel" in k for k in launched_kernels(lambda: h.sigma_device(x, y)))
    err = float((y.double() - ref).norm() / ref.norm())
    assert err <= 7e-8, err
    h.close()


@pytest.mark.parametrize("first", ["float64", "float32"])
def test_the_line_is_lower_for_fp32(first):
    """Sampled strings at a ratio of 18.5 multiply-adds to the direct kernel's: FP64 takes the rows kernel (1.2 times
    as fast), FP32, whose vectors pay FP64 products too, the direct one -- whichever asks first."""
    import torch

    import sbd_tpb
    import synth
    h1, eri, core = synth.synthetic_hamiltonian(20)
    s = synth.sample_strings(20, 6, 2800)
    prob = sbd_tpb.Problem(norb=20, nelec=12, core=core, h1=h1, eri_packed=eri, astr=s, bstr=s.copy())
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    x = torch.from_numpy(np.random.default_rng(1).normal(size=prob.ndet)).cuda()
    out = {}
    for dtype in (first, "float32" if first == "float64" else "float64"):
        v = x.to(getattr(torch, dtype))
        out[dtype] = torch.zeros_like(v)
        ran = launched_kernels(lambda: h.sigma_device(v, out[dtype]))
        assert any(("ab_rows" if dtype == "float64" else "ab_sparse") in k for k in ran), ran
    # FP32: vectors and results rounded to FP32, 2^-24 a value over a few thousand terms of random sign
    diff = (out["float32"].double() - out["float64"]).abs().max() / out["float64"].abs().max()
    assert float(diff) <= 2e-6
    h.close()
