"""Walled scenes whose wall data sits where the per-group wall codes, the tile
edges and the plate's halo faces meet: sparse face fractions anywhere in the
grid, with and without solid cells and a plate at a k tile's edge, on both step
kernels against the oracle, bit for bit (fields, plate, samples)."""
import dataclasses

import numpy as np
import pytest

from conftest import bits_equal, first_mismatch
from scenes import body_scene, drive_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch


def sparse_fractions(shape, share, rng):
    out = []
    for ax in range(3):
        s = list(shape)
        s[ax] -= 1
        f = np.ones(s, np.float32)
        pick = rng.random(s) < share
        f[pick] = rng.choice(np.array([0.0, 0.3, 0.8], np.float32), size=int(pick.sum()))
        out.append(f.ravel())
    return tuple(out)


@pytest.mark.parametrize("kernel", ["fused", "two_pass"])
@pytest.mark.parametrize("share", [0.002, 0.3])
# the plate is five cells below the top: at the last cell of a 64-cell k tile,
# at the first of the next (its lower faces are the tile below's), one further;
# and an odd room with one cell in its last group of four
@pytest.mark.parametrize("dims", [(24, 20, 68), (26, 19, 69), (24, 20, 70), (23, 37, 33)])
def test_sparse_walls_match_oracle(cuda, dims, share, kernel):
    from oracle import OracleFDTD
    from spectral_analyzer_b200 import AcousticFDTD
    sc = body_scene(*dims, seed=8)
    sc = dataclasses.replace(sc, fracs=sparse_fractions(dims, share, np.random.default_rng(5)))
    f, o = AcousticFDTD(**sc.kwargs()), OracleFDTD(**sc.kwargs())
    f.set_kernel(kernel)
    a, b = drive_scene(f, sc, 60), drive_scene(o, sc, 60)
    assert np.abs(b["P"]).max() > 0 and np.abs(b["W"]).max() > 0
    for k in b:
        x, y = np.ascontiguousarray(a[k]), np.ascontiguousarray(b[k])
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (k, first_mismatch(x, y) if x.dtype == np.float32 else k)


@pytest.mark.parametrize("kernel", ["fused", "two_pass"])
@pytest.mark.parametrize("dims", [(20, 33, 65), (17, 30, 31)])
def test_fractions_on_an_open_room_match_oracle(cuda, dims, kernel):
    """No solid cell and no plate; a second set of fractions replaces the first."""
    from oracle import OracleFDTD
    from spectral_analyzer_b200 import AcousticFDTD
    rng = np.random.default_rng(1)
    kw = dict(Nx=dims[0], Ny=dims[1], Nz=dims[2], dx=0.01, c=343.0, rho_air=1.21,
              cell_type=np.zeros(int(np.prod(dims)), np.uint8), plate_iz=-1,
              plate_active=np.zeros(dims[0] * dims[1], np.uint8), n_pml=4)
    f, o = AcousticFDTD(**kw), OracleFDTD(**kw)
    f.set_kernel(kernel)
    src = dims[2] // 2 + dims[2] * (dims[1] // 2 + dims[1] * (dims[0] // 2))
    for fr in (sparse_fractions(dims, 0.01, rng), sparse_fractions(dims, 0.2, rng)):
        for s in (f, o):
            s.set_face_fractions(*fr)
            s.add_pressure(src, 1.0)
            for _ in range(25):
                s.step(1)
        for name in ("get_pressure_field", "get_velocity_x", "get_velocity_y", "get_velocity_z"):
            x, y = np.asarray(getattr(f, name)()).ravel(), np.asarray(getattr(o, name)()).ravel()
            assert bits_equal(x, y), (name, first_mismatch(x, y))
