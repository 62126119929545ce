"""Rooms with more planes (or rows) than a grid has rows of blocks (65535): they
step on the single pass, whose grid counts tiles and segments, whichever kernel
their size alone would choose; walled ones get their wall codes and 16-bit ones
their pressure back.  Bit for bit against the oracle, or the room's own traces."""
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


# open: of a size that takes the two passes when it is not this long; walled:
# below and above the number of cells from which the single pass is automatic
@pytest.mark.parametrize("dims,wall,kernel", [
    ((70000, 4, 4), False, "auto"), ((65536, 3, 5), False, "auto"), ((66000, 4, 4), True, "fused"),
    ((66000, 4, 4), True, "auto"), ((70000, 8, 8), True, "auto"),
])
def test_more_planes_than_rows_of_blocks(cuda, dims, wall, kernel):
    from oracle import OracleFDTD
    from spectral_analyzer_b200 import AcousticFDTD
    nx, ny, nz = dims
    flat = lambda i, j, k: k + nz * (j + ny * i)
    ct = np.zeros(nx * ny * nz, np.uint8)
    if wall:
        ct[[flat(3, 1, 1), flat(65534, 2, 3), flat(nx - 4, 1, 2)]] = 1
    kw = dict(Nx=nx, Ny=ny, Nz=nz, dx=0.01, c=343.0, rho_air=1.21, cell_type=ct, plate_iz=-1,
              plate_active=np.zeros(nx * ny, np.uint8), n_pml=2)
    f, o = AcousticFDTD(**kw), OracleFDTD(**kw)
    f.set_kernel(kernel)
    for s in (f, o):
        for i in (5, 65533, nx - 6):
            s.add_pressure(flat(i, 1, 2), 1.0 + i % 3)
        for _ in range(3):
            s.step(1)
    f.step(4)
    for _ in range(4):
        o.step(1)
    for name in ("get_pressure_field", "get_velocity_x", "get_velocity_y", "get_velocity_z"):
        x, y = np.asarray(getattr(f, name)()).ravel(), np.asarray(getattr(o, name)()).ravel()
        assert np.abs(y[-ny * nz * 40:]).max() > 0 and bits_equal(x, y), (name, first_mismatch(x, y))


@pytest.mark.parametrize("dims", [(70000, 4, 5), (3, 530000, 4)])
@pytest.mark.parametrize("mode", ["bf16", "fp16c"])
def test_16bit_pressure_of_a_long_room(cuda, dims, mode):
    from spectral_analyzer_b200.precision import PrecisionRoom
    room = seeded_room(*dims, 8, seed=3, n_rec=1, n_pml=1, source_kind="gaussian")
    axis = int(np.argmax(dims))
    room.src = tuple(d - 2 if a == axis else 1 for a, d in enumerate(dims))
    room.sigma_steps = 1.0
    room.receivers = [tuple(d - 1 - q if a == axis else 1 + q % 2 for a, d in enumerate(dims)) for q in range(8)]
    r = PrecisionRoom(room, mode)
    r.step(8)
    p, last = r.pressure().reshape(dims), r.traces()[-1]
    assert np.abs(last).max() > 0                       # a tap of weight 1 and seven of weight 0
    assert np.array_equal([p[c] for c in room.receivers], last)
    r.close()
