"""The single-pass march by its own name (set_kernel "march"), one launch a step
whatever the room's size, bit for bit against the two-pass kernels (which deposit
and record with kernels of their own): its in-kernel source deposit and receiver
record at the edges of both tile shapes, and rooms of every automatic choice.
Launch counts show which kernels ran."""
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


def run(room, kernel, calls):
    from spectral_analyzer_b200 import AcousticFDTD
    f = AcousticFDTD(room.nx, room.ny, room.nz, room.dx, room.c, room.rho, cell_type=room.cell_type(),
                     plate_iz=-1, plate_active=room.plate_active(), n_pml=room.n_pml)
    f.set_face_absorption(room.absorption)
    f.set_kernel(kernel)
    assert f.kernel == kernel or kernel == "auto"
    f.set_point_source(room.src_flat, room.signal())
    f.set_receivers(*f.precompute_pressure_samplers(room.receiver_xyz()), sum(calls))
    launches = []
    for n in calls:
        l0 = f.launch_count
        f.step(n)
        launches.append(f.launch_count - l0)
    out = (f.get_traces(), f.get_pressure_field(), f.get_velocity_x(), f.get_velocity_y(), f.get_velocity_z())
    f.close()
    return out, launches


def compare(got, ref, what):
    assert np.abs(ref[0][:, 0]).max() > 0, what
    for name, a, b in zip(("traces", "P", "Vx", "Vy", "Vz"), got, ref):
        assert bits_equal(a, b), (what, name, first_mismatch(a, b))


# source cells on the edges of the tiles the march picks: 8 x 128, then 16 x 64
CASES = [
    ((24, 20, 256), [(12, 7, 127), (12, 8, 128), (12, 15, 129), (12, 16, 0), (0, 0, 0), (23, 19, 255), (5, 9, 124), (6, 10, 131)]),
    ((20, 36, 160), [(10, 15, 63), (10, 16, 64), (10, 31, 127), (10, 32, 128), (0, 35, 159), (19, 0, 60), (9, 13, 67), (11, 19, 3)]),
]


@pytest.mark.parametrize("dims,sources", CASES)
def test_source_and_record_on_tile_edges(cuda, dims, sources):
    from spectral_analyzer_b200.rooms import seeded_room
    calls = (1, 7, 1, 21)                               # records both in-kernel and flushed
    for q, src in enumerate(sources):
        room = seeded_room(*dims, 30, seed=40 + q, n_rec=3, n_pml=3, source_kind="gaussian")
        room.src = src
        room.receivers[0] = tuple(min(max(c + 2, 0), d - 1) for c, d in zip(src, dims))
        got, launches = run(room, "march", calls)
        ref, _ = run(room, "two_pass", calls)
        assert launches == [n + 1 for n in calls]       # a step's kernel each, and the last step's record
        compare(got, ref, src)


@pytest.mark.parametrize("dims", [(64, 64, 64), (73, 74, 75), (74, 73, 80), (97, 81, 65), (113, 111, 109)])
def test_rooms_of_every_automatic_choice(cuda, dims):
    from spectral_analyzer_b200.rooms import seeded_room
    room = seeded_room(*dims, 40, seed=sum(dims), n_rec=4, n_pml=5, source_kind="gaussian")
    room.receivers[0] = tuple(c + 2 for c in room.src)
    calls = (1, 11, 28)
    got, launches = run(room, "march", calls)
    ref, two = run(room, "two_pass", calls)
    assert launches == [n + 1 for n in calls] and min(two) > 2
    compare(got, ref, dims)
    auto, launches = run(room, "auto", calls)
    on_chip = np.prod(dims) < 1.2e6
    assert launches[1:] == ([2, 2] if on_chip else [2 * n + 1 for n in calls[1:]])
    compare(auto, ref, dims)
