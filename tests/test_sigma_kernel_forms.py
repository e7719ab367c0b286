"""Every kernel form of sigma gives the same bits (needs a B200).

Vectors whose rows are 16-byte aligned (row length a multiple of 16 bytes / element size, base
address 16-byte aligned) take the passes that cover two 16-byte column groups per thread; a vector
viewed one element into its buffer takes passes with scalar loads, per row or by distinct ket of 8 rows;
small problems one row per thread.  All sum the same terms in the same order with the same roundings (fused multiply-add for the doubles terms, rounded
FP64 products for the singles and the diagonal), so sigma is bitwise equal: general form
(convention 1, with and without accumulate) and exchange-symmetric one-pass form (convention 2)."""
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


def _vec(n, dtype, seed, symmetric):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=g)
    if symmetric:
        r = (r + r.T) * 0.5
    return r.to(dtype).reshape(-1).contiguous()


def _offset_copy(v):
    """v copied into a buffer one element longer and viewed from its second element: same values,
    contiguous, but not 16-byte aligned."""
    import torch
    buf = torch.empty(v.numel() + 1, dtype=v.dtype, device=v.device)
    view = buf[1:]
    view.copy_(v)
    assert view.data_ptr() % 16 != 0
    return view


# name -> norb, electrons and strings of each spin, and the same-spin passes that aligned and offset vectors
# take: one row per thread below 8,192 determinants per SM whatever the rows; with few connections the
# per-row passes of two column groups and of scalar loads; and a set between the lines of the two kinds of
# row (1.77 doubles per distinct ket, six CTAs of the per-row passes on an SM in FP64, eight in FP32), whose
# offset vectors take the union passes.
FORMS = {
    "fci12": (12, 6, 924, "sigma_block_kernel", "sigma_block_kernel"),
    "sci24": (24, 8, 1500, "_cm_kernel", "sigma_block_kernel"),
    "sci20": (20, 6, 2000, "_cm_kernel", "sigma_union_kernel"),
}


def _sampled(norb, n, count):
    import synth
    from sbd_tpb import Problem
    h1, eri, core = synth.synthetic_hamiltonian(norb)
    s = synth.sample_strings(norb, n, count)
    return Problem(norb=norb, nelec=2 * n, core=core, h1=h1, eri_packed=eri, astr=s, bstr=s.copy())


def _passes(names):
    """The same-spin passes among kernel names."""
    return [k for k in names if "sigma_" in k and "_kernel" in k and "sigma_sym_add" not in k]


@pytest.mark.parametrize("name", sorted(FORMS))
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_aligned_and_offset_vectors_give_same_bits(name, dtype):
    import torch

    import sbd_tpb
    norb, ne, count, aligned, offset = FORMS[name]
    prob = _sampled(norb, ne, count)
    tdt = getattr(torch, dtype)
    n = len(prob.astr)
    assert n % (16 // torch.empty(0, dtype=tdt).element_size()) == 0  # aligned rows
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    for symmetric in (False, True):
        x = _vec(n, tdt, 5, symmetric)
        y0 = _vec(n, tdt, 6, False)
        for accumulate in ((False,) if symmetric else (False, True)):
            a_out, u_out, u_x = y0.clone(), _offset_copy(y0), _offset_copy(x)
            for want, xx, yy in ((aligned, x, a_out), (offset, u_x, u_out)):
                ran = _passes(launched_kernels(
                    lambda: h.sigma_device(xx, yy, accumulate=accumulate, symmetric=symmetric)))
                assert len(ran) == (1 if symmetric else 2) and all(want in k for k in ran), ran
            assert torch.isfinite(a_out).all()
            assert torch.equal(a_out, u_out), (name, dtype, symmetric, accumulate,
                                               float((a_out.double() - u_out.double()).abs().max()))
    h.close()


@pytest.mark.parametrize("norb, ne, count, dtype, union", [
    (20, 6, 2000, "float64", False),  # sampled, 1.77 doubles per distinct ket, six per-row CTAs on an SM
    (20, 6, 2000, "float32", False),
    (20, 6, 2001, "float64", True),   # scalar rows
    (22, 7, 4000, "float32", False),  # 1.58
    (24, 8, 1500, "float64", False),  # 1.29
    (24, 8, 1501, "float32", False),
])
def test_union_passes_on_sampled_sets(norb, ne, count, dtype, union):
    """On sampled sets the per-row passes with 16-byte rows stay ahead well above 1.5 doubles per distinct
    ket (20 orbitals, 2,000 strings: FP64 0.39 against 0.46 ms, FP32 0.23 against 0.36)."""
    import torch

    import sbd_tpb
    prob = _sampled(norb, ne, count)
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    x = _vec(count, getattr(torch, dtype), 5, True)
    y = torch.empty_like(x)
    for symmetric in (False, True):
        ran = _passes(launched_kernels(lambda: h.sigma_device(x, y, symmetric=symmetric)))
        assert ran and all(("sigma_union_kernel" in k) == union for k in ran), ran
    h.close()


@pytest.mark.parametrize("norb, ne, na, nb, dtype, symmetric, alpha, beta", [
    # a grid of 2.4 CTAs an SM: FP32 union passes from 1.6 doubles per distinct ket (0.34 against 0.44 ms)
    (21, 5, 1444, 1020, "float32", False, True, True),
    (20, 6, 1200, 1200, "float64", False, True, True),  # 5.1 CTAs an SM, 1.7 doubles per distinct ket
    # beta's 14,000 rows of 100 columns: threads of a union tile idle (FP32 2.0 against 2.6 ms at 30,000)
    (20, 6, 100, 14000, "float32", False, False, False),
    (20, 6, 100, 14000, "float64", False, False, True),
    # one-pass FP32 at 2.4 doubles per distinct ket: 0.26 against 0.30 ms
    (18, 7, 1200, 1200, "float32", True, False, None),
    (18, 7, 1200, 1200, "float64", True, True, None),
])
def test_union_passes_on_rectangular_and_one_pass(norb, ne, na, nb, dtype, symmetric, alpha, beta):
    import torch

    import sbd_tpb
    import synth
    from test_ab_rows import _dense
    h1, eri, core = synth.synthetic_hamiltonian(norb)
    strings = [synth.sample_strings(norb, ne, n) if (norb, ne) == (20, 6) else _dense(norb, ne, n, 1) for n in (na, nb)]
    prob = sbd_tpb.Problem(norb=norb, nelec=2 * ne, core=core, h1=h1, eri_packed=eri, astr=strings[0], bstr=strings[1])
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    x = torch.randn(na, nb, dtype=getattr(torch, dtype), device="cuda")
    if symmetric:
        x = x + x.T
    x = x.reshape(-1).contiguous()
    y = torch.zeros_like(x)
    ran = ["union" in k for k in _passes(launched_kernels(lambda: h.sigma_device(x, y, symmetric=symmetric)))]
    assert ran == ([alpha] if symmetric else [alpha, beta])
    h.close()
