"""A scheduled source in a solid cell: its sample is shared among the open cells
beside it by a kernel of its own, after the receivers have heard the step before.
Receivers on those cells, on every step kernel against the oracle, bit for bit."""
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


@pytest.mark.parametrize("kernel", ["auto", "march", "fused", "two_pass"])
# on a face of the block (one open neighbour), an edge (two) and a corner (three)
@pytest.mark.parametrize("src", [(9, 12, 15), (9, 9, 15), (9, 9, 10)])
def test_receivers_beside_a_solid_source(cuda, src, kernel):
    from oracle import OracleFDTD
    from spectral_analyzer_b200 import AcousticFDTD
    dims = (22, 24, 31)
    ct = np.zeros(dims, np.uint8)
    ct[9:14, 9:17, 10:20] = 1
    kw = dict(Nx=dims[0], Ny=dims[1], Nz=dims[2], dx=0.01, c=343.0, rho_air=1.21, cell_type=ct.ravel(), plate_iz=-1,
              plate_active=np.zeros(dims[0] * dims[1], np.uint8), n_pml=4)
    f, o = AcousticFDTD(**kw), OracleFDTD(**kw)
    f.set_kernel(kernel)
    flat = src[2] + dims[2] * (src[1] + dims[1] * src[0])
    signal = np.random.default_rng(3).standard_normal(30).astype(np.float32)
    xyz = np.float32([[src[0] - 1, src[1], src[2]], [src[0] - 1.4, src[1] + 0.3, src[2] - 0.6], [4, 5, 6]])
    idx, w = o.precompute_pressure_samplers(xyz)
    f.set_point_source(flat, signal)
    f.set_receivers(idx, w, 40)
    for n in (1, 2, 17, 20):                           # the signal ends inside the last call
        f.step(n)
    ref = o.run(40, flat, signal, idx, w)
    got = f.get_traces()
    assert np.abs(ref[:, 0]).max() > 0
    assert bits_equal(got, ref), first_mismatch(got, ref)
    assert bits_equal(f.get_pressure_field(), o.get_pressure_field())
