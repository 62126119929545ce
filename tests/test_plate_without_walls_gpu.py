"""An active plate whose cells carry a code that is neither air nor solid: the
scene then has no solid cell, no face fractions and no mask, on both step kernels
against the oracle, bit for bit, with the plate at the last cell of a k tile, at
the first of the next (its lower faces are the tile below's) and inside one."""
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


@pytest.mark.parametrize("kernel", ["fused", "two_pass"])
@pytest.mark.parametrize("dims,iz", [((20, 18, 72), 63), ((20, 18, 72), 64), ((17, 21, 30), 11)])
def test_plate_of_unnamed_cells_matches_oracle(cuda, dims, iz, kernel):
    from oracle import OracleFDTD
    from spectral_analyzer_b200 import AcousticFDTD
    nx, ny, nz = dims
    ct = np.zeros(dims, np.uint8)
    ct[:, :, iz] = 7
    active = np.zeros((nx, ny), np.uint8)
    active[3:-3, 4:-4] = 1
    kw = dict(Nx=nx, Ny=ny, Nz=nz, dx=0.01, c=343.0, rho_air=1.21, cell_type=ct.ravel(), plate_iz=iz,
              plate_active=active.ravel(), n_pml=3)
    f, o = AcousticFDTD(**kw), OracleFDTD(**kw)
    f.set_kernel(kernel)
    force = np.int32([nx // 2 * ny + ny // 2, (nx // 2 + 1) * ny + ny // 2])
    for n in (1, 1, 2, 20):
        for s in (f, o):
            s.inject_plate_force(force, np.float32([0.6, 0.4]), 0.5)
            s.add_pressure(iz - 3 + nz * (ny // 2 + ny * (nx // 2)), 0.25)
        f.step(n)
        for _ in range(n):
            o.step(1)
    for name in ("get_pressure_field", "get_velocity_x", "get_velocity_y", "get_velocity_z", "get_plate_displacement"):
        x, y = np.asarray(getattr(f, name)()).ravel(), np.asarray(getattr(o, name)()).ravel()
        assert np.abs(y).max() > 0 and bits_equal(x, y), (name, first_mismatch(x, y))
