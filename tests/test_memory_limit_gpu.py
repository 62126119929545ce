"""A room whose second velocity set does not fit the device's memory: the step says
so, again at every try, and the handle steps on once there is room, with the
two-pass kernels' bits.  Through the C interface, whose handles own their fields."""
import ctypes as C

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


def ptr(a, t):
    return a.ctypes.data_as(C.POINTER(t))


def create(lib, dims):
    ct, pa = np.zeros(int(np.prod(dims)), np.uint8), np.zeros(dims[0] * dims[1], np.uint8)
    h = lib.fdtd_create(*dims, 0.01, 343.0, 1.21, ptr(ct, C.c_uint8), -1, ptr(pa, C.c_uint8), 7.0, 0.45, 2.0, 1e-5, 6)
    assert h
    return C.c_void_p(h)


def pressure(lib, h, dims):
    out = np.empty(int(np.prod(dims)), np.float32)
    assert lib.fdtd_get_pressure_field(h, ptr(out, C.c_float), out.size) == 0
    return out


@pytest.mark.parametrize("kernel", [0, 3])              # the march either way: 16.8M cells
def test_second_velocity_set_without_room(cuda, kernel):
    from spectral_analyzer_b200 import _native
    lib = _native.load()
    dims = (256, 256, 256)
    field = 4 * int(np.prod(dims))
    a, b, warm = create(lib, dims), create(lib, dims), create(lib, (160, 128, 96))
    for h in (a, b, warm):
        assert lib.fdtd_b200_add_pressure(h, (dims[0] // 4) * 128 * 96, 1.0) == 1
    lib.fdtd_b200_set_kernel(a, kernel)
    lib.fdtd_b200_set_kernel(b, 1)
    lib.fdtd_b200_set_kernel(warm, 3)
    assert lib.fdtd_step(warm, 2) == 0                  # the kernel is loaded before memory is short
    cuda.cuda.empty_cache()
    free = cuda.cuda.mem_get_info()[0]
    rest = cuda.empty((free - field - field // 2 >> 21 << 21,), dtype=cuda.uint8, device="cuda")   # 1.5 fields left
    for _ in range(3):
        assert lib.fdtd_step(a, 1) == _native.FDTD_ERR_CUDA
        assert "out of memory" in _native.last_error()
    assert lib.fdtd_get_step_count(a) == 0
    del rest
    cuda.cuda.empty_cache()
    for h in (a, b):
        assert lib.fdtd_step(h, 12) == 0
    x, y = pressure(lib, a, dims), pressure(lib, b, dims)
    assert np.abs(y).max() > 0 and bits_equal(x, y), first_mismatch(x, y)
    for h in (a, b, warm):
        lib.fdtd_destroy(h)


def test_scheduled_source_without_room(cuda):
    """The sample of a step that found no memory is deposited when the step is taken."""
    from spectral_analyzer_b200 import _native
    lib = _native.load()
    dims = (256, 256, 256)
    field = 4 * int(np.prod(dims))
    a, b, warm = create(lib, dims), create(lib, dims), create(lib, (160, 128, 96))
    signal = np.float32([1.0, 0.5, -0.25])
    for h in (a, b):
        assert lib.fdtd_b200_set_point_source(h, (dims[0] // 4) * 256 * 256 + 9000, ptr(signal, C.c_float), 3) == 0
    lib.fdtd_b200_set_kernel(b, 1)
    lib.fdtd_b200_set_kernel(warm, 3)
    assert lib.fdtd_step(warm, 2) == 0
    cuda.cuda.empty_cache()
    free = cuda.cuda.mem_get_info()[0]
    rest = cuda.empty((free - field - field // 2 >> 21 << 21,), dtype=cuda.uint8, device="cuda")
    for _ in range(2):
        assert lib.fdtd_step(a, 1) == _native.FDTD_ERR_CUDA
    del rest
    cuda.cuda.empty_cache()
    for h in (a, b):
        assert lib.fdtd_step(h, 5) == 0
    x, y = pressure(lib, a, dims), pressure(lib, b, dims)
    assert np.abs(y).max() > 0 and bits_equal(x, y), first_mismatch(x, y)
    for h in (a, b, warm):
        lib.fdtd_destroy(h)


@pytest.mark.parametrize("mode", ["bf16", "fp16c", "fp64"])
def test_pressure_is_read_in_parts_when_memory_is_short(cuda, mode):
    from spectral_analyzer_b200.precision import PrecisionRoom
    from spectral_analyzer_b200.rooms import seeded_room
    room = seeded_room(250, 251, 253, 6, seed=2, n_rec=1, n_pml=4, source_kind="gaussian")
    room.sigma_steps = 1.0
    whole, parts = PrecisionRoom(room, mode), PrecisionRoom(room, mode)
    for r in (whole, parts):
        r.step(6)
    ref = whole.pressure()                              # 15.9M values at once
    whole.close()
    cuda.cuda.empty_cache()
    free = cuda.cuda.mem_get_info()[0]
    rest = cuda.empty((free - (40 << 20) >> 21 << 21,), dtype=cuda.uint8, device="cuda")
    got = parts.pressure()                              # in 40 MB
    del rest
    cuda.cuda.empty_cache()
    parts.close()
    assert np.abs(ref).max() > 0 and np.array_equal(got.view(np.uint64), ref.view(np.uint64))
