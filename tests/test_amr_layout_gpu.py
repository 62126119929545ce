"""The AMR step's device layouts on irregular topologies, bit for bit against a
plain NumPy float32 restatement: cells with no face and with more faces than
the kernel fetches ahead, counts that are no multiple of a warp or of four,
wall cells, order-8 grids whose stencil rows are too many to be numbered, and
the nearest-cell search with ties, closed cells and no candidate."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C, RHO, DX = 343.0, 1.21, 0.01


@pytest.fixture(scope="module")
def cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for -m gpu tests")
    return torch


def graph(n_cells, n_faces, seed):
    rng = np.random.default_rng(seed)
    neg = rng.integers(0, n_cells - 1, n_faces)
    neg[: n_faces // 8] = rng.integers(0, 5, n_faces // 8)            # a few cells with very many faces
    pos = (neg + rng.integers(1, n_cells - 1, n_faces)) % (n_cells - 1)   # the last cell has none
    pos = np.where(pos == neg, (neg + 1) % (n_cells - 1), pos)
    types = rng.choice(np.array([0, 0, 0, 3, 1, 2], np.uint8), n_cells)
    types[-1] = 0
    return {"centers": rng.uniform(0, 1, (n_cells, 3)), "vol": rng.uniform(0.5, 1.5, n_cells) * DX ** 3,
            "open": rng.choice([1.0, 0.5, 0.25], n_cells), "types": types, "neg": neg.astype(np.int32),
            "pos": pos.astype(np.int32), "area": rng.uniform(0.5, 1.0, n_faces) * DX * DX * 0.05,
            "fopen": rng.choice([1.0, 0.75], n_faces), "dist": rng.uniform(1.0, 2.0, n_faces) * DX}


def solver(g, order):
    from spectral_analyzer_b200.amr import AcousticAMR
    return AcousticAMR(g["centers"], g["vol"], g["open"], g["types"], g["neg"], g["pos"], g["area"], g["fopen"],
                       g["dist"], C, RHO, DX, order)


def reference(g, order, dt, p, steps):
    f = np.float32
    p, v = p.copy(), np.zeros(len(g["neg"]), f)
    dt_rho, bulk = f(f(dt) / f(RHO)), f(RHO * C * C * dt)
    flux = (g["area"] * g["fopen"]).astype(f)
    inv = f(1.0) / g["dist"].astype(f)
    acoustic = ((g["types"] == 0) | (g["types"] == 3)) & (g["open"] > 0)
    inv_den = np.where(acoustic, 1.0 / (g["vol"] * g["open"]), 0.0).astype(f)
    zero = (g["types"] == 1) | (g["types"] == 2)
    neg, pos = g["neg"], g["pos"]
    one = f(1.0)
    for _ in range(steps):
        if order == 2:
            grad = (p[pos] - p[neg]) * inv
        else:   # four slots on each side, unused ones reading cell 0 with weight 0
            z = f(0.0) * p[0]
            grad = (f(0.0) + -inv * p[neg]) + z + z + z
            grad = grad + inv * p[pos] + z + z + z
        v = (v - dt_rho * grad) * one
        d = np.zeros(len(p), f)
        for q in range(len(neg)):
            d[neg[q]] = d[neg[q]] + flux[q] * v[q]
            d[pos[q]] = d[pos[q]] + -flux[q] * v[q]
        p = p * one - ((bulk * d) * inv_den) * one
        p[zero] = 0.0
    return p, v


@pytest.mark.parametrize("n_cells,n_faces,order", [(1003, 3001, 2), (31, 66, 2), (70, 129, 8), (20011, 70003, 8)])
def test_irregular_topology(cuda, n_cells, n_faces, order):
    g = graph(n_cells, n_faces, n_cells)
    s = solver(g, order)
    p = np.zeros(n_cells, np.float32)
    for c in (0, 3, n_cells - 2):
        if g["types"][c] in (0, 3):
            s.inject_pressure_nearest(g["centers"][c], 0.5 + c % 7)
            p[c] += np.float32(0.5 + c % 7)
    assert np.array_equal(s.get_pressure(), p)
    steps = 3
    assert s.step(steps) == 0
    want_p, want_v = reference(g, order, s.dt, p, steps)
    assert np.array_equal(s.get_velocity().view(np.uint32), want_v.view(np.uint32))
    assert np.array_equal(s.get_pressure().view(np.uint32), want_p.view(np.uint32))
    s.close()


def test_nearest_cell(cuda):
    g = graph(600, 900, 5)
    g["types"][:] = 0
    g["centers"][:] = np.random.default_rng(1).uniform(2, 3, (600, 3))
    g["centers"][[37, 412]] = [0.25, 0.5, 0.5], [0.75, 0.5, 0.5]      # equally far from the middle
    g["centers"][100] = [0.5, 0.5, 0.5]
    g["types"][100] = 1                                               # the nearest one is a wall
    s = solver(g, 2)
    s.inject_pressure_nearest([0.5, 0.5, 0.5], 2.0)
    s.inject_pressure_nearest([0.76, 0.5, 0.5], 3.0)
    p = s.get_pressure()
    assert p[37] == 2.0 and p[412] == 3.0 and np.count_nonzero(p) == 2
    for bad in ([np.nan, 0.5, 0.5], [1e200, 0.0, 0.0]):
        with pytest.raises(RuntimeError, match="rc=-2"):
            s.inject_pressure_nearest(bad, 1.0)
    assert np.array_equal(s.get_pressure(), p)
    s.close()
