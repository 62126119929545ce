"""Open rooms of the sizes whose steps are taken in two passes, against the single
pass (set_kernel "fused"), bit for bit: fields and traces, with the source beside
the room's faces and at the ends of a group of four cells, a signal that ends
before the run, none at all, a receiver on the source cell, and steps one at a
time and many at a time."""
import numpy as np
import pytest

from conftest import bits_equal, first_mismatch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch


def make(dims, kernel, src, sig, xyz):
    from spectral_analyzer_b200 import AcousticFDTD
    f = AcousticFDTD(*dims, 0.01, 343.0, 1.21, cell_type=np.zeros(int(np.prod(dims)), np.uint8), plate_iz=-1,
                     plate_active=np.zeros(dims[0] * dims[1], np.uint8), n_pml=5)
    f.set_kernel(kernel)
    f.set_receivers(*f.precompute_pressure_samplers(xyz), 40)
    f.add_pressure((dims[0] // 2 * dims[1] + dims[1] // 2) * dims[2] + dims[2] // 2, 1.0)
    if sig is not None:
        f.set_point_source((src[0] * dims[1] + src[1]) * dims[2] + src[2], sig)
    return f


@pytest.mark.parametrize("dims", [(73, 74, 75), (74, 73, 80), (113, 111, 109), (90, 128, 120)])
@pytest.mark.parametrize("n_sig", [None, 7, 40])
def test_open_two_pass_equals_single_pass(cuda, dims, n_sig):
    sig = None if n_sig is None else np.linspace(1.0, -2.0, n_sig).astype(np.float32)
    hi = tuple(d - 1 for d in dims)
    for src in [(0, 0, 0), hi, (1, dims[1] - 2, 4), (dims[0] // 2, 2, dims[2] - 2), (dims[0] // 2 + 1, dims[1] // 2, 35)]:
        xyz = np.array([src, (dims[0] / 2 + 1.3, dims[1] / 2 - 1.6, dims[2] / 2 + 0.4)], np.float32)
        a, b = (make(dims, k, src, sig, xyz) for k in ("auto", "fused"))
        for f in (a, b):
            f.step(1)
            f.step_async(1)
            assert f.synchronize() == 0
            f.step(11)
            f.step(1)
        assert a.step_count == b.step_count == 14
        for name in ("get_pressure_field", "get_velocity_x", "get_velocity_y", "get_velocity_z", "get_traces"):
            x, y = getattr(a, name)(), getattr(b, name)()
            assert np.abs(y).max() > 0 and bits_equal(x, y), (src, name, first_mismatch(x, y))
        if sig is None:
            break
