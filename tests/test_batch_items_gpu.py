"""The batch's own choice of tile shape and item depth: members of one set after
another, whose best shapes differ, keep their single-room results bit for bit,
with captured graphs and without."""
import numpy as np
import pytest

from conftest import bits_equal, first_mismatch

pytestmark = pytest.mark.gpu

# (rooms of the set): a flat one, one wide row of cells, uneven mixes
SETS = [[(40, 24, 60)], [(24, 16, 256), (9, 8, 128)], [(33, 40, 48), (5, 9, 130), (64, 17, 33)], [(1, 30, 70), (70, 1, 20)]]


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch


def rooms(dims, steps):
    from spectral_analyzer_b200.rooms import seeded_room
    out = []
    for q, d in enumerate(dims):
        r = seeded_room(*d, steps, seed=50 + q, n_rec=3, n_pml=3, source_kind="gaussian")
        r.src = tuple(min(c + 1, n - 1) for c, n in zip(r.receivers[0], d))
        out.append(r)
    return out


@pytest.mark.parametrize("graph", [True, False])
def test_sets_of_differing_shapes(cuda, graph):
    from spectral_analyzer_b200.serving import EngineBatch, make_solver
    b = EngineBatch()
    steps = 24
    for dims in SETS + SETS[::-1]:
        rs = rooms(dims, steps)
        got = [make_solver(r) for r in rs]
        b.set(got, [steps] * len(got))
        b.step(8, graph)
        b.step(8, graph)
        b.step(8, graph)
        done, status = b.sync()
        assert list(done) == [steps] * len(got) and not status.any()
        b.set([], [])
        for r, f in zip(rs, got):
            ref = make_solver(r)
            ref.set_kernel("two_pass")
            ref.step(steps)
            t = ref.get_traces()
            assert np.abs(t).max() > 0
            assert bits_equal(f.get_traces(), t)
            a, c = f.get_pressure_field(), ref.get_pressure_field()
            assert bits_equal(a, c), first_mismatch(a, c)
            ref.close()
            f.close()
