"""The adjoint sweeps where their layout can go wrong: rows that end inside a
group of four cells, a receiver on the source cell (recorded without the next
step's sample), a signal shorter than the run, and segments of one, several and
all steps.  The float forward is the float oracle bit for bit; the double
gradient is torch.autograd's of the same model to 1e-9 (both sum the same double
terms, in other orders: some 1e5 of them, 1e5 * 2^-53 = 1e-11 of the largest)."""
import numpy as np
import pytest

from spectral_analyzer_b200.adjoint import differentiation_problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch


def problem(n, steps, seed):
    p = differentiation_problem(n, n_steps=steps, seed=seed, n_rec=3, n_pml=4, corr=3.0)
    p.receivers[1] = p.src
    return p


@pytest.mark.parametrize("n", [(17, 15, 21), (14, 18, 22), (15, 14, 27), (16, 33, 64)])
@pytest.mark.parametrize("n_sig", [70, 30, 1])
def test_forward_records_before_the_next_sample(cuda, n, n_sig):
    from oracle import OracleFDTD
    from spectral_analyzer_b200 import _native
    from spectral_analyzer_b200.adjoint import AdjointRoom
    prob = problem(n, 70, 4)
    r = AdjointRoom(prob)
    sig = np.ascontiguousarray(1.0 + prob.signal()[:n_sig], np.float64)
    assert r._lib.fdtd_b200_adj_set_source(r._h, prob.flat(prob.src), sig.ctypes.data_as(_native.P_f64), sig.size) == 0
    r.set_absorption(prob.a)
    y = r.forward()
    nx, ny, nz = prob.shape
    o = OracleFDTD(nx, ny, nz, prob.dx, prob.c, prob.rho, n_pml=prob.n_pml)
    o.set_cell_absorption(prob.a)
    idx, w = r.taps
    ref = o.run(prob.n_steps, prob.flat(prob.src), sig, idx, w.astype(np.float32))
    assert np.abs(ref).max() > 0
    assert np.array_equal(y.astype(np.float32).view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("every", [1, 17, 60])
@pytest.mark.parametrize("n", [(17, 15, 21), (14, 18, 22)])
def test_double_gradient_is_torch_autograd(cuda, n, every):
    from spectral_analyzer_b200.adjoint import AdjointRoom
    from torch_reference import loss_and_grad
    prob = problem(n, 60, 6)
    tgt = np.random.default_rng(2).standard_normal((prob.n_steps, len(prob.receivers)))
    r = AdjointRoom(prob, double=True, checkpoint_every=every)
    r.set_absorption(prob.a)
    y = r.forward()
    g = r.backward(2.0 * (y - tgt))
    loss, ref = loss_and_grad(prob.a, prob, *r.taps, tgt, device="cuda", segment=30)
    assert float(np.sum((y - tgt) ** 2)) == pytest.approx(loss, rel=1e-12)
    assert np.linalg.norm(ref) > 0 and np.linalg.norm(g - ref) <= 1e-9 * np.linalg.norm(ref)
