"""The 16-bit single pass adds its source sample in shared memory, in every CTA
whose box holds the source cell and in no other: bit for bit against the two-pass
kernels (which add it in memory), with sources in the first planes of a march
(whose halo planes have negative numbers), at the ends of segments and on the
edges of both tile shapes, and on the steps after the signal has ended."""
import numpy as np
import pytest

from spectral_analyzer_b200.rooms import seeded_room

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch


# (grid, sources): 16 x 64 tiles, then 8 x 128 tiles
CASES = [
    ((30, 36, 60), [(0, 0, 0), (1, 15, 59), (2, 16, 7), (29, 35, 8)]),
    ((24, 20, 200), [(0, 7, 127), (1, 8, 128), (2, 0, 199), (3, 19, 120), (23, 4, 136)]),
]


@pytest.mark.parametrize("mode", ("bf16", "fp16", "bf16c", "fp16c"))
@pytest.mark.parametrize("dims,sources", CASES)
def test_source_in_the_first_planes_and_on_tile_edges(cuda, mode, dims, sources):
    from spectral_analyzer_b200.precision import PrecisionRoom
    for q, src in enumerate(sources):
        room = seeded_room(*dims, 12, seed=60 + q, n_rec=2, n_pml=2, source_kind="gaussian")
        room.src, room.sigma_steps = src, 1.0
        room.receivers[0] = tuple(min(c + 2, d - 1) for c, d in zip(src, dims))
        outs = []
        for kernel in ("fused", "two_pass"):
            r = PrecisionRoom(room, mode, kernel=kernel, trace_capacity=20)
            r.step(5)
            r.step(15)                      # the signal has 12 samples
            outs.append((r.pressure(), r.traces()))
            r.close()
        assert np.abs(outs[1][1][:, 0]).max() > 0, src
        for a, b in zip(*outs):
            assert np.array_equal(a.view(np.uint64), b.view(np.uint64)), (mode, dims, src)
