"""Handles whose buffers do not fit the device's memory: the call says so, at every
try, no other call reports it again, and the handle steps on once there is room."""
import ctypes as C

import numpy as np
import pytest

from conftest import bits_equal, first_mismatch
from spectral_analyzer_b200.rooms import seeded_room

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


@pytest.mark.parametrize("mode", ["fp16", "bf16c"])
def test_second_16_bit_velocity_set_without_room(cuda, mode):
    from spectral_analyzer_b200.precision import PrecisionRoom
    room = seeded_room(250, 251, 253, 8, seed=2, n_rec=2, n_pml=4, source_kind="gaussian")
    room.receivers[0] = tuple(c + 2 for c in room.src)
    ref, got = PrecisionRoom(room, mode), PrecisionRoom(room, mode)
    ref.step(8)
    field = 2 * 250 * 251 * 256
    rest = only(cuda, 2 * field + field // 2)           # of three or six
    for _ in range(2):
        with pytest.raises(RuntimeError, match="memory"):
            got.step(8)
    del rest
    cuda.cuda.empty_cache()
    got.step(8)
    assert np.abs(ref.traces()).max() > 0
    assert np.array_equal(got.traces().view(np.uint64), ref.traces().view(np.uint64))
    assert np.array_equal(got.pressure().view(np.uint64), ref.pressure().view(np.uint64))


@pytest.mark.parametrize("kernel", ["fused", "two_pass"])
def test_steps_after_receivers_did_not_fit(cuda, kernel):
    from spectral_analyzer_b200 import _native
    from spectral_analyzer_b200.precision import PrecisionRoom
    room = seeded_room(30, 36, 60, 20, seed=4, n_rec=4, n_pml=3, source_kind="gaussian")
    ref, got = (PrecisionRoom(room, "bf16", kernel=kernel) for _ in range(2))
    idx, w = np.tile(got._idx, 64), np.tile(got._w, 64)
    rc = got._lib.fdtd_b200_prec_set_receivers(got._h, idx.size // 8, idx.ctypes.data_as(_native.P_i32),
                                               w.ctypes.data_as(_native.P_f64), 2 ** 31 - 1, 0)   # 4 TB of traces
    assert rc == _native.FDTD_ERR_CUDA and "memory" in _native.last_error()
    for r in (ref, got):
        r.step(20)
    assert np.abs(ref.pressure()).max() > 0
    assert np.array_equal(got.pressure().view(np.uint64), ref.pressure().view(np.uint64))


def test_slab_steps_after_receivers_did_not_fit(cuda):
    from spectral_analyzer_b200 import _native
    from spectral_analyzer_b200.slab import local_room
    room = seeded_room(20, 21, 44, 20, seed=4, n_rec=2, n_pml=3, source_kind="gaussian")
    ref, got = local_room(room, 1, fused=True), local_room(room, 1, fused=True)
    lib, h = _native.load(), got.slabs[0]._h
    idx, w = np.zeros(8 * 256, np.int32), np.ones(8 * 256, np.float32)
    rc = lib.fdtd_b200_slab_set_receivers(h, 256, idx.ctypes.data_as(_native.P_i32), w.ctypes.data_as(_native.P_f32),
                                          2 ** 31 - 1)                                             # 2 TB of traces
    assert rc == _native.FDTD_ERR_CUDA and "memory" in _native.last_error()
    for r in (ref, got):
        r.step(20)
    assert np.abs(ref.pressure_field()).max() > 0 and bits_equal(got.pressure_field(), ref.pressure_field())


def test_other_handles_step_after_a_room_that_did_not_fit(cuda):
    from spectral_analyzer_b200 import AcousticFDTD, _native
    room = seeded_room(64, 60, 68, 20, seed=5, n_rec=2, n_pml=4, source_kind="gaussian")
    lib, dims = _native.load(), (256, 256, 256)
    outs = []
    for fail in (False, True):
        f = AcousticFDTD(room.nx, room.ny, room.nz, room.dx, room.c, room.rho, cell_type=room.cell_type(), plate_iz=-1,
                         plate_active=room.plate_active(), n_pml=room.n_pml)
        f.set_kernel("march")
        f.set_point_source(room.src_flat, room.signal())
        f.step(1)
        if fail:
            rest = only(cuda, 3 * 4 * 256 ** 3)         # of five fields
            ct, pa = np.zeros(256 ** 3, np.uint8), np.zeros(256 ** 2, np.uint8)
            u8 = C.POINTER(C.c_uint8)
            assert not lib.fdtd_create(*dims, 0.01, 343.0, 1.21, ct.ctypes.data_as(u8), -1, pa.ctypes.data_as(u8), 7.0,
                                       0.45, 2.0, 1e-5, 6)
            assert "memory" in _native.last_error()
        f.step(19)
        outs.append(f.get_pressure_field())
    del rest
    cuda.cuda.empty_cache()
    assert np.abs(outs[0]).max() > 0 and bits_equal(*outs), first_mismatch(*outs)


@pytest.mark.parametrize("graph", [0, 1])
def test_batch_set_that_does_not_fit_leaves_no_members(cuda, graph):
    """The set's first room is in order, its second finds no memory for its second
    velocity set: the batch then steps nothing, and the first room goes on alone."""
    from spectral_analyzer_b200 import _native
    lib = _native.load()

    def create(dims, kernel):
        ct, pa = np.zeros(int(np.prod(dims)), np.uint8), np.zeros(dims[0] * dims[1], np.uint8)
        u8 = C.POINTER(C.c_uint8)
        h = C.c_void_p(lib.fdtd_create(*dims, 0.01, 343.0, 1.21, ct.ctypes.data_as(u8), -1, pa.ctypes.data_as(u8), 7.0,
                                       0.45, 2.0, 1e-5, 4))
        sig = np.float32([1.0, 0.5, 0.25, -1.0, 2.0, 0.125, 1.5, -0.5] * 5)
        cell = dims[2] // 2 + dims[2] * (dims[1] // 2 + dims[1] * (dims[0] // 2))
        assert h.value and lib.fdtd_b200_set_point_source(h, cell, sig.ctypes.data_as(_native.P_f32), sig.size) == 0
        assert lib.fdtd_b200_set_kernel(h, kernel) == 0
        return h

    def pressure(h, dims):
        out = np.empty(int(np.prod(dims)), np.float32)
        assert lib.fdtd_get_pressure_field(h, out.ctypes.data_as(_native.P_f32), out.size) == 0
        return out

    small, large = (40, 36, 44), (256, 256, 256)
    a, big, ref, ref_big = create(small, 3), create(large, 0), create(small, 1), create(large, 1)
    b = C.c_void_p(lib.fdtd_b200_batch_create(0))
    members = (C.c_void_p * 2)(a, big)
    limits = np.int32([40, 8])
    lim = limits.ctypes.data_as(C.POINTER(C.c_int))
    assert lib.fdtd_step(a, 1) == 0                     # its second set is there
    assert lib.fdtd_b200_batch_set(b, members, lim, 1) == 0 and lib.fdtd_b200_batch_step(b, 4, graph) == 0
    rest = only(cuda, 4 * 256 ** 3 * 3 // 2)            # one field of three and a half
    for _ in range(2):
        assert lib.fdtd_b200_batch_set(b, members, lim, 2) == _native.FDTD_ERR_CUDA
        assert "memory" in _native.last_error()
        assert lib.fdtd_get_step_count(a) == 5
        l0 = lib.fdtd_b200_batch_launch_count(b)
        assert lib.fdtd_b200_batch_step(b, 4, graph) == 0 and lib.fdtd_b200_batch_launch_count(b) == l0
        assert lib.fdtd_b200_batch_sync(b, None, None) == 0 and lib.fdtd_get_step_count(a) == 5
    assert lib.fdtd_step(a, 4) == 0                     # alone, its next sample deposited once
    del rest
    cuda.cuda.empty_cache()
    assert lib.fdtd_b200_batch_set(b, members, lim, 2) == 0
    assert lib.fdtd_b200_batch_step(b, 40, graph) == 0 and lib.fdtd_b200_batch_sync(b, None, None) == 0
    assert lib.fdtd_get_step_count(a) == 40 and lib.fdtd_get_step_count(big) == 8
    assert lib.fdtd_b200_batch_set(b, None, None, 0) == 0
    for h, g, dims, n in ((a, ref, small, 40), (big, ref_big, large, 8)):
        assert lib.fdtd_step(g, n) == 0
        x, y = pressure(h, dims), pressure(g, dims)
        assert np.abs(y).max() > 0 and bits_equal(x, y), first_mismatch(x, y)
    lib.fdtd_b200_batch_destroy(b)
    for h in (a, big, ref, ref_big):
        lib.fdtd_destroy(h)
