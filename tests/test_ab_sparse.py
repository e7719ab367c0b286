"""The direct alpha-beta kernel (csrc/sigma.cu, ab_sparse_kernel) against the oracle, in both of its forms: the beta
program in one range of kets, and split by ket range where a string has more than a few singles but too few
for the rows kernel (sampled sets, the products 20 to 100 times the direct loop's multiply-adds)."""
import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norb, ne, na, nb, ranges", [
    (22, 7, 4000, 4000, True),    # 7 singles a string
    (22, 7, 3001, 2500, True),    # unequal lists, odd rows
    (24, 8, 2000, 2000, False),   # 1.4 singles a string
])
def test_direct_kernel_against_oracle(norb, ne, na, nb, ranges):
    import pyoracle
    import torch

    import sbd_tpb
    import synth
    h1, eri, core = synth.synthetic_hamiltonian(norb, seed=5)
    prob = sbd_tpb.Problem(norb=norb, nelec=2 * ne, core=core, h1=h1, eri_packed=eri,
                           astr=synth.sample_strings(norb, ne, na), bstr=synth.sample_strings(norb, ne, nb))
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    rng = np.random.default_rng(7)
    x = rng.normal(size=prob.ndet)
    rows = np.sort(rng.choice(prob.ndet, size=200, replace=False)).astype(np.uint64)
    ham = pyoracle.Hamiltonian.from_arrays(norb, prob.nelec, core, h1, eri)
    ref = pyoracle.System(ham, prob.astr, prob.bstr).sigma_rows(rows, x)
    scale = float(np.max(np.abs(ref)))
    idx = torch.from_numpy(rows.astype(np.int64)).cuda()
    # FP64 sums of the same terms in another order; FP32 vectors, sums and results, 2^-24 a value
    for dtype, tol in (("float64", 1e-12), ("float32", 2e-6)):
        v = torch.from_numpy(x).cuda().to(getattr(torch, dtype))
        y = torch.zeros_like(v)
        ran = [k for k in launched_kernels(lambda: h.sigma_device(v, y, separated=False)) if "ab_sparse_kernel" in k]
        # template arguments: type, staged rows, ket ranges
        assert len(ran) == 1 and ran[0].split("<")[1].split(">")[0].split(",")[2].strip() == str(ranges).lower(), ran
        assert float(np.max(np.abs(y[idx].double().cpu().numpy() - ref))) <= tol * scale, dtype
    if na == nb:
        g = torch.Generator(device="cuda").manual_seed(3)
        r = torch.randn(na, nb, dtype=torch.float64, device="cuda", generator=g)
        s = (r + r.T).reshape(-1).contiguous()
        gen, sym = torch.zeros_like(s), torch.zeros_like(s)
        h.sigma_device(s, gen)
        h.sigma_device(s, sym, symmetric=True)
        assert float((sym - gen).abs().max()) <= 1e-13 * float(gen.abs().max())
    h.close()
