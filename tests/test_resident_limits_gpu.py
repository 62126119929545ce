"""Small rooms whose many-step launch cannot be had or does not finish: the calls
step on the other kernels, or report a timeout, and the handle runs on."""
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


def solver(room, kernel, capacity):
    from spectral_analyzer_b200 import AcousticFDTD
    f = AcousticFDTD(room.nx, room.ny, room.nz, room.dx, room.c, room.rho, cell_type=room.cell_type(), plate_iz=-1,
                     plate_active=room.plate_active(), n_pml=room.n_pml)
    f.set_kernel(kernel)
    f.set_point_source(room.src_flat, room.signal())
    f.set_receivers(*f.precompute_pressure_samplers(room.receiver_xyz()), capacity)
    return f


def near_room(dims, steps, seed):
    room = seeded_room(*dims, steps, seed=seed, n_rec=3, n_pml=4, source_kind="gaussian")
    room.receivers[0] = tuple(c + 2 for c in room.src)
    return room


def same(f, g):
    tr = f.get_traces(), g.get_traces()
    assert np.abs(tr[1]).max() > 0 and bits_equal(*tr)
    for name in ("get_pressure_field", "get_velocity_x", "get_velocity_y", "get_velocity_z"):
        x, y = getattr(f, name)(), getattr(g, name)()
        assert bits_equal(x, y), (name, first_mismatch(x, y))


@pytest.mark.parametrize("dims", [(40, 36, 44), (96, 80, 72)])   # then the march, and the two passes
@pytest.mark.parametrize("asynchronous", [False, True])
def test_refused_launch_steps_on_the_other_kernels(cuda, dims, asynchronous):
    room = near_room(dims, 40, 7)
    f, g = solver(room, "auto", 60), solver(room, "two_pass", 60)
    f.step(9)                                          # one launch and its receivers' rows
    assert f.launch_count == 2
    f.debug_refuse_resident()
    for n in (20, 3, 28):
        l0 = f.launch_count
        (f.step_async if asynchronous else f.step)(n)
        assert f.launch_count - l0 > n
    assert f.synchronize() == 0
    g.step(60)
    same(f, g)


def test_async_steps_do_not_wait_when_receivers_grow(cuda):
    """More receivers than before, then steps queued behind work that is still running."""
    room = near_room((40, 36, 44), 30, 8)
    f, g = solver(room, "auto", 60), solver(room, "two_pass", 60)
    f.step(10)
    g.step(10)
    rng = np.random.default_rng(0)
    xyz = np.concatenate([room.receiver_xyz(), rng.uniform(0, 30, (100, 3)).astype(np.float32)])
    for h in (f, g):
        h.set_receivers(*h.precompute_pressure_samplers(xyz), 60)
    done = cuda.cuda.Event()
    with cuda.cuda.stream(f.torch_stream()):
        cuda.cuda._sleep(1_000_000_000)                # half a second
        done.record()
    f.step_async(30)
    assert not done.query()
    assert f.synchronize() == 0
    g.step(30)
    same(f, g)


@pytest.mark.parametrize("dims,brick", [((64, 64, 64), 0), ((65, 57, 61), 17), ((96, 80, 72), 5)])
def test_timed_out_exchange_is_reported_and_recovered(cuda, dims, brick):
    """A brick that publishes nothing: every block gives up after its bounded wait
    (a few milliseconds) and the kernel ends by itself; the handle steps on after a reset."""
    from spectral_analyzer_b200 import _native
    room = near_room(dims, 30, 9)
    f, g = solver(room, "auto", 200), solver(room, "two_pass", 200)
    f.step(6)
    assert f.synchronize() == 0                        # no hold: no timeout
    f.debug_hold_brick(brick, wait_us=3000)
    l0 = f.launch_count
    f.step_async(12)
    with pytest.raises(RuntimeError, match="timed out"):
        f.synchronize()
    assert f.launch_count - l0 == 2 and "timed out" in _native.last_error()
    f.debug_hold_brick(-1)
    f.step_async(3)                                    # the latch holds until reset
    with pytest.raises(RuntimeError, match="timed out"):
        f.synchronize()
    cuda.cuda.synchronize()                            # the context is fine
    f.reset()
    assert f.synchronize() == 0
    for n in (1, 25, 34):
        f.step(n)
    g.step(60)
    assert f.synchronize() == 0
    same(f, g)


def test_brick_hook_rejects_bad_arguments(cuda):
    room = near_room((40, 36, 44), 5, 10)
    f = solver(room, "auto", 10)
    for brick, wait_us in ((-2, 0), (1 << 20, 0), (0, -1), (0, 1 << 30)):
        with pytest.raises(ValueError):
            f.debug_hold_brick(brick, wait_us)
    f.step(3)
    assert f.synchronize() == 0
    big = solver(near_room((160, 128, 112), 5, 10), "auto", 10)     # does not fit the chip
    with pytest.raises(ValueError):
        big.debug_hold_brick(0)


def test_small_rooms_on_their_own_streams_at_once(cuda):
    """Three rooms whose launches need their blocks resident together, queued at the
    same time from one thread and from three, as each steps alone."""
    import threading
    rooms = [near_room(d, 60, 11) for d in ((64, 64, 64), (96, 80, 72), (33, 41, 29))]
    fs, gs = ([solver(r, k, 400) for r in rooms] for k in ("auto", "two_pass"))
    for _ in range(5):
        for f in fs:
            f.step_async(20)
    def drive(f):
        for n in (100, 37, 63):
            f.step(n)
    threads = [threading.Thread(target=drive, args=(f,)) for f in fs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for f, g in zip(fs, gs):
        assert f.synchronize() == 0 and f.step_count == 300
        g.step(300)
        same(f, g)
