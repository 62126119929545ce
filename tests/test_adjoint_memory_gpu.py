"""An adjoint handle whose checkpoints, segment states or fields do not fit the
device's memory: the call says so, again at every try, and the handle gives the
same gradient once there is room.  Receivers that do not fit leave a handle whose
forward is refused."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch


def only(torch, left):
    """Takes the device's memory but for about `left` bytes."""
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    return torch.empty((free - left >> 21 << 21,), dtype=torch.uint8, device="cuda")


def test_gradient_after_memory_ran_short(cuda):
    from spectral_analyzer_b200.adjoint import AdjointRoom, differentiation_problem
    prob = differentiation_problem(160, n_steps=24, seed=3)
    prob.receivers[0] = tuple(c + 2 for c in prob.src)  # reached within the run
    field = 4 * 160 ** 3
    resid = np.random.default_rng(1).standard_normal((24, len(prob.receivers)))
    a, b = AdjointRoom(prob, checkpoint_every=8), AdjointRoom(prob, checkpoint_every=8)
    a.set_absorption(prob.a)
    b.set_absorption(prob.a)
    traces = a.forward()
    ref = a.backward(resid)
    a.close()
    rest = only(cuda, 6 * field)                        # three checkpoints of four fields do not fit
    for _ in range(2):
        with pytest.raises(RuntimeError, match="memory"):
            b.forward()
    del rest
    cuda.cuda.empty_cache()
    assert np.array_equal(b.forward(), traces)
    rest = only(cuda, (4 * 9 + 3) * field)              # the states of a segment do, the sweep's fields not
    for _ in range(2):
        with pytest.raises(RuntimeError, match="memory"):
            b.backward(resid)
    del rest
    cuda.cuda.empty_cache()
    got = b.backward(resid)
    assert np.abs(ref).max() > 0 and np.array_equal(got.view(np.uint64), ref.view(np.uint64))
    b.close()


def test_forward_is_refused_after_receivers_did_not_fit(cuda):
    from spectral_analyzer_b200 import _native
    from spectral_analyzer_b200.adjoint import AdjointRoom, differentiation_problem
    prob = differentiation_problem(40, n_steps=10, seed=3)
    prob.receivers[0] = tuple(c + 1 for c in prob.src)
    room = AdjointRoom(prob)
    room.set_absorption(prob.a)
    traces = room.forward()
    idx, w = np.tile(room.taps[0].ravel(), 64), np.tile(room.taps[1].ravel(), 64)
    lib, p = _native.load(), (idx.ctypes.data_as(_native.P_i32), w.ctypes.data_as(_native.P_f64))
    rc = lib.fdtd_b200_adj_set_receivers(room._h, idx.size // 8, *p, 2 ** 31 - 1)    # 2 TB of traces
    assert rc == _native.FDTD_ERR_CUDA and "memory" in _native.last_error()
    with pytest.raises(RuntimeError):
        room.forward()
    assert lib.fdtd_b200_adj_set_receivers(room._h, room.n_rec, *p, 10) == 0
    assert np.abs(traces).max() > 0 and np.array_equal(room.forward(), traces)
    room.close()
