"""Small rooms stepped many steps per launch, bit for bit against the two-pass
kernels: grids at the edges of every compiled brick (a last brick of one plane,
row or cell; thin rooms; one brick only; one and several planes per thread),
calls that end inside and across the 256-step check, sources on brick corners
and receivers whose taps span bricks."""
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


def run(dims, kernel, calls, src, n_rec=3, n_pml=4, asynchronous=False):
    from spectral_analyzer_b200 import AcousticFDTD
    from spectral_analyzer_b200.rooms import gaussian_pulse, seeded_room
    room = seeded_room(*dims, sum(calls), seed=sum(dims), n_rec=n_rec, n_pml=n_pml)
    f = AcousticFDTD(*dims, room.dx, room.c, room.rho, cell_type=room.cell_type(), plate_iz=-1,
                     plate_active=room.plate_active(), n_pml=n_pml)
    f.set_face_absorption(room.absorption)
    f.set_kernel(kernel)
    xyz = room.receiver_xyz()
    xyz[0] = [min(c + 1, d - 1) - 0.4 for c, d in zip(src, dims)]     # eight taps around the source
    idx, w = f.precompute_pressure_samplers(xyz)
    f.set_point_source(room.flat(*src), gaussian_pulse(sum(calls) - 5, 5.0))
    f.set_receivers(idx, w, sum(calls) - 3)                           # the last rows do not fit
    launches = []
    for n in calls:
        l0 = f.launch_count
        if asynchronous:
            f.step_async(n)
        else:
            f.step(n)
        launches.append(f.launch_count - l0)
    assert f.synchronize() == 0
    out = (f.get_traces(), f.get_pressure_field(), f.get_velocity_x(), f.get_velocity_y(), f.get_velocity_z())
    f.close()
    return out, launches


# (grid, source)
CASES = [
    ((4, 8, 8), (3, 7, 7)), ((33, 41, 29), (2, 8, 8)), ((64, 64, 64), (15, 15, 15)), ((65, 57, 61), (16, 16, 32)),
    ((37, 9, 129), (9, 8, 64)), ((1, 40, 50), (0, 16, 31)), ((40, 1, 50), (3, 0, 32)), ((50, 40, 1), (20, 8, 0)),
    ((200, 30, 30), (100, 29, 0)), ((97, 81, 65), (12, 16, 33)), ((96, 96, 96), (47, 48, 63)), ((128, 96, 96), (16, 31, 32)),
]


@pytest.mark.parametrize("dims,src", CASES)
def test_many_steps_per_launch_equal_two_pass(cuda, dims, src):
    calls = (1, 2, 3, 60, 210)                        # the check falls inside the last call
    got, launches = run(dims, "fused", calls, src)
    ref, _ = run(dims, "two_pass", calls, src)
    assert launches[3] <= 2 and launches[4] <= 5      # one launch and its receivers' rows per window
    assert np.abs(ref[0][:, 0]).max() > 0
    for name, a, b in zip(("traces", "P", "Vx", "Vy", "Vz"), got, ref):
        assert bits_equal(a, b), (name, first_mismatch(a, b))


def test_async_windows_and_many_receivers(cuda):
    """step_async, and more taps than the kernel records (the march takes those steps)."""
    for n_rec, windowed in ((128, True), (129, False)):
        got, launches = run((48, 40, 36), "fused", (300,), (20, 16, 16), n_rec=n_rec, asynchronous=True)
        ref, _ = run((48, 40, 36), "two_pass", (300,), (20, 16, 16), n_rec=n_rec)
        assert (launches[0] < 20) == windowed
        for a, b in zip(got, ref):
            assert bits_equal(a, b), first_mismatch(a, b)


def test_reset_and_source_past_its_end(cuda):
    """A handle reset in mid-run starts over exactly; steps after the signal's end add nothing."""
    from spectral_analyzer_b200 import AcousticFDTD
    f = AcousticFDTD(45, 50, 55, 0.01, cell_type=np.zeros(45 * 50 * 55, np.uint8), plate_iz=-1,
                     plate_active=np.zeros(45 * 50, np.uint8), n_pml=5)
    f.set_point_source(20 + 55 * (25 + 50 * 22), np.float32([1.0, -0.5, 0.25]))
    outs = []
    for calls in ((40,), (1,) * 40):
        f.reset()
        for n in calls:
            f.step(n)
        outs.append((f.get_pressure_field(), f.get_velocity_y()))
    assert np.abs(outs[0][0]).max() > 0
    for a, b in zip(*outs):
        assert bits_equal(a, b), first_mismatch(a, b)
