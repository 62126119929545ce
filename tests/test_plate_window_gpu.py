"""Plate scenes stepped many steps per call (the plate guard read once per
window) against the same steps one call at a time, bit for bit on both step
kernels: fields, plate, traces, return codes and the state a failed plate
update in mid-window leaves behind."""
import numpy as np
import pytest

from conftest import bits_equal, first_mismatch
from scenes import body_scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch


def make(sc, kernel, capacity):
    from spectral_analyzer_b200 import AcousticFDTD
    f = AcousticFDTD(**sc.kwargs())
    f.set_face_fractions(*sc.fracs)
    f.set_kernel(kernel)
    f.set_bridge_sources(sc.bridge_idx, sc.bridge_wgt)
    f.set_receivers(*f.precompute_pressure_samplers(sc.rec_xyz), capacity)
    return f


def state(f):
    return {"P": f.get_pressure_field(), "Vx": f.get_velocity_x(), "Vy": f.get_velocity_y(), "Vz": f.get_velocity_z(),
            "W": f.get_plate_displacement(), "steps": f.step_count, "traces": f.get_traces()}


def same(a, b):
    for k in a:
        if k == "steps":
            assert a[k] == b[k]
        else:
            assert a[k].shape == b[k].shape and bits_equal(a[k], b[k]), (k, first_mismatch(a[k], b[k]))


@pytest.mark.parametrize("kernel", ["fused", "two_pass"])
@pytest.mark.parametrize("dims", [(24, 20, 16), (37, 29, 41)])
def test_window_equals_single_steps(cuda, kernel, dims):
    sc = body_scene(*dims, seed=3)
    a, b = make(sc, kernel, 290), make(sc, kernel, 290)
    src = sc.point_cells[0]
    for f in (a, b):
        f.set_point_source(src, np.float32([0.3, -0.2, 0.1]))      # the first steps go one at a time
    drive = np.full(sc.bridge_idx.size, 0.3, np.float32)
    for n in (1, 5, 90, 200):                                        # the last call crosses the 256-step check
        for f in (a, b):
            f.inject_bridge_drive(drive, 1.0)
            f.inject_plate_force(sc.force_idx, sc.force_wgt, 0.2)
        assert a.step_rc(n) == 0
        for _ in range(n):
            assert b.step_rc(1) == 0
    x, y = state(a), state(b)
    assert np.abs(y["W"]).max() > 0 and np.abs(y["traces"]).max() > 0
    same(x, y)


@pytest.mark.parametrize("kernel", ["fused", "two_pass"])
def test_plate_fails_in_mid_window(cuda, kernel):
    sc = body_scene(seed=2)
    a, b = make(sc, kernel, 80), make(sc, kernel, 80)
    rc, amp = [], 4e3
    while len(rc) in (0, 80):                                        # the least push that ends within 80 steps
        amp *= 1.25
        drive = np.full(sc.bridge_idx.size, amp, np.float32)
        b.reset()
        b.inject_bridge_drive(drive, 1.0)
        rc = [b.step_rc(1)]
        while rc[-1] == 0 and len(rc) < 80:
            rc.append(b.step_rc(1))
    assert rc[-1] == -3 and len(rc) > 1                              # some steps pass first
    a.inject_bridge_drive(drive, 1.0)
    assert a.step_rc(80) == -3
    same(state(a), state(b))
    for f in (a, b):                                                 # it fails there again, changing nothing
        assert f.step_rc(4) == -3
    same(state(a), state(b))
    for f in (a, b):                                                 # a failing step keeps its pending forces
        f.reset()
        f.inject_bridge_drive(1e4 * drive, 1.0)
        assert f.step_rc(7) == -3 and f.step_count == 0
        f.inject_bridge_drive(-1e4 * drive, 1.0)
        f.inject_bridge_drive(0.01 * drive, 1.0)
        assert f.step_rc(3) == 0
    same(state(a), state(b))
