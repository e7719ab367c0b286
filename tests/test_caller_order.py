"""Calls on device buffers wait for the work that the caller queued on the default stream before them: each
buffer is filled behind a kernel that keeps the stream busy for some tens of milliseconds, and the call
follows without a synchronisation."""
import numpy as np
import pytest

from conftest import golden_problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def problem():
    import torch

    import sbd_tpb
    prob, _, _ = golden_problem("syn10_ab")
    h = sbd_tpb.Handle(0)
    h.set_problem(prob)
    x = torch.from_numpy(np.random.default_rng(3).normal(size=prob.ndet)).cuda()
    x /= x.norm()
    yield h, x
    h.close()


def _late(buf, value):
    """buf := value, behind a busy default stream."""
    import torch
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)
    buf.copy_(value) if hasattr(value, "shape") else buf.fill_(value)
    return buf


def _rdm(h, x):
    import sbd_tpb
    L = h.problem.norb
    one, two = np.zeros(2 * L ** 2), np.zeros(4 * L ** 4)
    sbd_tpb._check(sbd_tpb.lib().sbd_tpb_rdm(h.h, x.data_ptr(), one.ctypes.data, two.ctypes.data, sbd_tpb.DEVICE))
    return np.concatenate([one, two])


def _sigma(call):
    def run(h, x):
        import torch
        y = torch.zeros_like(x)
        getattr(h, call)(x, y)
        torch.cuda.synchronize()
        return y.cpu().numpy()
    return run


def _carryover(h, x):
    import sbd_tpb
    r = h.carryover(x, sbd_tpb.CARRYOVER_CUTOFF_SINGLES, threshold=1e-4, mem=sbd_tpb.DEVICE)
    return np.concatenate([r["astr"], r["bstr"], [r["total_weight"]]]).astype(np.float64)


@pytest.mark.parametrize("call", [_sigma("sigma"), _sigma("sigma_device"), _sigma("sigma_noalloc"), _rdm, _carryover],
                         ids=["sigma", "sigma_device", "sigma_noalloc", "rdm", "carryover"])
def test_input_written_just_before_the_call(problem, call):
    import torch
    h, x = problem
    ref = call(h, x)
    buf = torch.zeros_like(x)
    # the RDMs' mixed term is summed with atomics: the last digits depend on their order
    assert np.allclose(call(h, _late(buf, x)), ref, rtol=0, atol=1e-13)


def test_output_buffer_still_in_use(problem):
    """A buffer that queued work still writes (as a caching allocator hands them out) is written after it."""
    import torch

    import sbd_tpb
    h, x = problem
    buf = torch.zeros_like(x)
    sbd_tpb._check(sbd_tpb.lib().sbd_tpb_diagonal(h.h, _late(buf, 7.0).data_ptr(), sbd_tpb.DEVICE))
    torch.cuda.synchronize()
    assert np.array_equal(buf.cpu().numpy(), h.diagonal())


def test_noalloc_under_capture(problem):
    """While the handle's stream is capturing nothing is waited for (a wait on work outside the graph would end
    the capture); replays read the input as it then is."""
    import torch
    h, x = problem
    buf, y = torch.zeros_like(x), torch.zeros_like(x)
    h.sigma_noalloc(x, y)
    torch.cuda.synchronize()
    ref = y.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.ExternalStream(h.stream())):
        h.sigma_noalloc(buf, y)
    buf.copy_(x)
    y.zero_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ref)
    del g
