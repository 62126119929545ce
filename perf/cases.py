"""The engine's everyday work as timed cases.

Each case is one pass a program makes through the package's public entry
points: a block of live ticks, a room run from its source to its traces, a
serving chunk of mixed rooms, a co-evolver's substeps, a walled scene, a room
stored in 16 bits, an absorption gradient and AMR steps.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what the program holds before the pass
    run(state)           one pass; its outputs, whole
    work(case)           bytes and operations the pass cannot do without
    exact(case, seed)    the same outputs from plain float64 torch
"""
import math

import numpy as np
import torch

from spectral_analyzer_b200 import AcousticFDTD
from spectral_analyzer_b200.adjoint import AdjointRoom, DiffProblem, boundary_absorption, trace_loss
from spectral_analyzer_b200.amr import AcousticAMR
from spectral_analyzer_b200.precision import PrecisionRoom
from spectral_analyzer_b200.rooms import gaussian_pulse, seeded_room
from spectral_analyzer_b200.serving import EngineBatch, make_solver

DX, C0, RHO = 0.01, 343.0, 1.21
SERVING_AXES = tuple(range(32, 257, 16))   # the axes serving requests are drawn from
CELL_FLOPS = 40                            # separately rounded operations of one cell-update
STORAGE = {"bf16": 2, "fp16": 2, "bf16c": 4, "fp16c": 4}


def listed():
    return [
        # a live caller: one source sample in, one step, the microphones out, per tick
        {"name": "live_64", "kind": "live", "nx": 64, "ny": 64, "nz": 64, "steps": 64, "rec": 8},
        # the small golden room, as a study runs it over and over
        {"name": "room_64", "kind": "room", "nx": 64, "ny": 64, "nz": 64, "steps": 400, "rec": 1, "n_pml": 10,
         "absorption": 0.1, "filled": False},
        # odd sizes: no axis a multiple of a tile or of the row padding
        {"name": "room_ragged", "kind": "room", "nx": 109, "ny": 87, "nz": 61, "steps": 300, "rec": 4, "n_pml": 8,
         "absorption": 0.3, "filled": False},
        # an ordinary serving-sized room on its own
        {"name": "room_mid", "kind": "room", "nx": 160, "ny": 128, "nz": 112, "steps": 200, "rec": 4, "n_pml": 10,
         "absorption": 0.15, "filled": False},
        # the largest room, its air already moving
        {"name": "room_large", "kind": "room", "nx": 512, "ny": 384, "nz": 256, "steps": 40, "rec": 8, "n_pml": 10,
         "absorption": 0.15, "filled": True},
        # one chunk of the continuous-batching server over mixed rooms
        {"name": "serve_mix", "kind": "serve", "rooms": 8, "steps": 64, "mix": 21},
        # the co-evolver around a guitar-sized body: plate drive, step, saddle samples per substep
        {"name": "body_substeps", "kind": "substeps", "nx": 170, "ny": 140, "nz": 74, "steps": 48},
        # a walled scene with a plate that no longer fits the caches
        {"name": "body_large", "kind": "body", "nx": 256, "ny": 200, "nz": 128, "steps": 64},
        # a room whose fields are stored in 16 bits, stepped on and its pressure read back
        {"name": "storage_bf16", "kind": "storage", "nx": 224, "ny": 160, "nz": 160, "steps": 400, "mode": "bf16"},
        # the gradient of a receiver loss with respect to the absorption field
        {"name": "gradient_128", "kind": "gradient", "nx": 128, "ny": 128, "nz": 128, "steps": 256, "every": 200},
        # AMR, second order, two refinement levels
        {"name": "amr_levels", "kind": "amr", "n": 52, "fine": 24, "order": 2, "steps": 256},
        # AMR, eighth order
        {"name": "amr_order8", "kind": "amr", "n": 72, "fine": 0, "order": 8, "steps": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("live", "room", "room", "room", "serve", "substeps", "body", "storage", "gradient", "amr"))
    if kind == "live":
        return {"kind": kind, "nx": _log(rng, 32, 128), "ny": _log(rng, 32, 128), "nz": _log(rng, 32, 128),
                "steps": rng.randint(16, 64), "rec": rng.randint(1, 8)}
    if kind == "room":
        while True:
            nx, ny, nz = _log(rng, 30, 512), _log(rng, 30, 384), _log(rng, 30, 384)
            if nx * ny * nz <= 40_000_000:
                break
        steps = max(24, min(400, int(1.5e9 / (nx * ny * nz))))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(steps // 2, steps),
                "rec": rng.randint(1, 8), "n_pml": rng.randint(4, 12), "absorption": round(rng.uniform(0.02, 1.0), 3),
                "filled": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": kind, "rooms": rng.randint(3, 8), "steps": rng.randint(24, 64), "mix": rng.randint(1, 10 ** 6)}
    if kind == "substeps":
        return {"kind": kind, "nx": rng.randint(90, 180), "ny": rng.randint(80, 150), "nz": rng.randint(34, 80),
                "steps": rng.randint(16, 48)}
    if kind == "body":
        return {"kind": kind, "nx": _log(rng, 100, 300), "ny": _log(rng, 100, 240), "nz": _log(rng, 40, 160),
                "steps": rng.randint(24, 64)}
    if kind == "storage":
        return {"kind": kind, "nx": _log(rng, 64, 224), "ny": _log(rng, 64, 160), "nz": _log(rng, 64, 160),
                "steps": rng.randint(160, 400), "mode": rng.choice(sorted(STORAGE))}
    if kind == "gradient":
        return {"kind": kind, "nx": rng.randint(32, 128), "ny": rng.randint(32, 128), "nz": rng.randint(32, 128),
                "steps": rng.randint(64, 256), "every": rng.choice((50, 100, 200))}
    order = rng.choice((2, 8))
    n = rng.randint(30, 60 if order == 2 else 72)
    return {"kind": "amr", "n": n, "fine": rng.randint(8, n // 2) if order == 2 else 0, "order": order,
            "steps": rng.randint(48, 192)}


# ------------------------------------------------------------------- inputs
def _room(case, seed):
    """A room with a seeded source cell, receivers and per-face absorption around the case's value."""
    r = seeded_room(case["nx"], case["ny"], case["nz"], case["steps"], seed=seed, n_rec=case["rec"],
                    source_kind="gaussian", n_pml=case["n_pml"])
    rng = np.random.default_rng(seed + 7)
    a = case["absorption"]
    r.absorption = tuple(float(v) for v in (a * rng.uniform(0.6, 1.0, 6)).astype(np.float32))
    r.sigma_steps = 8.0
    near = r.receivers[0]   # the first receiver close enough to hear the source within the pass
    r.src = tuple(int(min(max(n + d, 0), m - 1)) for n, d, m in zip(near, (6, -4, 5), (r.nx, r.ny, r.nz)))
    return r


def _solver(r):
    f = AcousticFDTD(r.nx, r.ny, r.nz, r.dx, r.c, r.rho, cell_type=r.cell_type(), plate_iz=-1,
                     plate_active=r.plate_active(), n_pml=r.n_pml)
    f.set_face_absorption(r.absorption)
    return f


def _moving_air(shape, seed):
    """A smooth random pressure field (a sum of plane waves, about 0.1 Pa), float32 on the GPU."""
    rng = np.random.default_rng(seed + 11)
    axes = [torch.arange(n, dtype=torch.float32, device="cuda") for n in shape]
    p = torch.zeros(shape, dtype=torch.float32, device="cuda")
    for _ in range(4):
        k = rng.uniform(0.1, 0.6, 3)
        ph = rng.uniform(0, 2 * math.pi, 3)
        w = [torch.sin(float(k[a]) * axes[a] + float(ph[a])) for a in range(3)]
        p += 0.1 * w[0][:, None, None] * w[1][None, :, None] * w[2][None, None, :]
    return p


def _serve_rooms(case, seed):
    shapes = np.random.default_rng(case["mix"])
    rng = np.random.default_rng(seed + 3)
    rooms = []
    for q in range(case["rooms"]):
        nx, ny, nz = (int(shapes.choice(SERVING_AXES)) for _ in range(3))
        r = seeded_room(nx, ny, nz, case["steps"], seed=int(rng.integers(1 << 30)), n_rec=int(shapes.integers(1, 5)),
                        source_kind="gaussian" if q % 2 else "ricker")
        r.f0, r.sigma_steps = 3000.0, 5.0
        near = r.receivers[0]
        r.src = tuple(int(min(max(n + d, 0), m - 1)) for n, d, m in zip(near, (5, -3, 4), (nx, ny, nz)))
        rooms.append(r)
    return rooms


def _body(nx, ny, nz, seed):
    """A closed instrument body: back, ribs, a plate with a soundhole, cut-cell
    fractions on the faces beside solid cells, a bridge and a neck force."""
    rng = np.random.default_rng(seed)
    back, piz = 3, nz - 6
    ii, jj = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    ci, cj, ri, rj = (nx - 1) / 2.0, (ny - 1) / 2.0, nx * 0.32, ny * 0.32
    inside = ((ii - ci) / ri) ** 2 + ((jj - cj) / rj) ** 2 < 1.0
    rib = ~inside & (np.abs(ii - ci) < ri + 2) & (np.abs(jj - cj) < rj + 2)
    hole = (ii - ci) ** 2 + (jj - (cj + rj * 0.35)) ** 2 < (0.08 * nx) ** 2
    ct = np.zeros((nx, ny, nz), np.uint8)
    ct[:, :, back:piz + 1][rib] = 1
    ct[:, :, back][inside] = 1
    active = inside & ~hole
    ct[:, :, piz][active] = 2
    solid = ct > 0
    fr = []
    for ax in range(3):
        n = ct.shape[ax]
        a, b = solid.take(range(n - 1), ax), solid.take(range(1, n), ax)
        f = np.where(a | b, 0.0, 1.0).astype(np.float32)
        bd = a ^ b
        f[bd] = rng.choice(np.array([0.0, 0.25, 0.5, 0.75], np.float32), size=int(bd.sum()))
        fr.append(f)
    fr[2][:, :, piz - 1][active] = 1.0
    fr[2][:, :, piz][active] = 1.0
    bi, bj = int(ci), int(cj - rj * 0.4)
    w = np.exp(-((ii - bi) ** 2 + (jj - bj) ** 2) / (2 * 1.5 ** 2))
    bridge = np.argwhere((w >= 1e-3) & active)
    b_idx = (piz - 1 + nz * (bridge[:, 1] + ny * bridge[:, 0])).astype(np.int32)
    nodes = np.argwhere(active)
    pick = nodes[np.sort(rng.choice(len(nodes), 10, replace=False))]
    flat = (pick[:, 1] + ny * pick[:, 0]).astype(np.int32)
    return {"ct": ct, "active": active, "piz": piz, "fr": fr, "b_idx": b_idx,
            "b_w": w[active & (w >= 1e-3)].astype(np.float32), "b_node": bridge[:, 1] + ny * bridge[:, 0],
            "f_idx": flat[:2].copy(), "f_w": np.float32([0.6, 0.4]), "s_idx": flat[2:].copy(),
            "s_w": np.full(8, 0.25, np.float32)}


def _drives(case, b, seed):
    """Bridge drives and neck forces of every substep: a pluck of seeded shape."""
    rng = np.random.default_rng(seed + 5)
    shape = rng.uniform(0.5, 1.5, b["b_idx"].size)
    t = np.arange(case["steps"])
    d = 0.05 * np.exp(-t / 60.0) * np.sin(2 * math.pi * t / 23.0 + rng.uniform(0, 1))
    return (d[:, None] * shape[None, :]).astype(np.float32), (0.02 * np.cos(t / 11.0)).astype(np.float32)


BODY_DX = 0.004   # grid spacing of the instrument bodies


def _body_solver(case, b):
    f = AcousticFDTD(case["nx"], case["ny"], case["nz"], BODY_DX, C0, RHO, cell_type=b["ct"].ravel(),
                     plate_iz=b["piz"], plate_active=b["active"].astype(np.uint8).ravel(), n_pml=6)
    f.set_face_fractions(*[x.ravel() for x in b["fr"]])
    f.set_bridge_sources(b["b_idx"], b["b_w"])
    return f


def _storage_room(case, seed):
    c = dict(case, rec=4, n_pml=10, absorption=0.15)
    return _room(c, seed)


def _gradient_problem(case, seed):
    rng = np.random.default_rng(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    n_pml = 10
    inner = lambda: tuple(int(rng.integers(n_pml + 1, d - n_pml - 1)) for d in shape)  # noqa: E731
    src = inner()
    recs = [tuple(int(min(max(s + d, 0), n - 1)) for s, d, n in zip(src, (4, 3, -5), shape))] + [inner() for _ in range(3)]
    a = boundary_absorption(shape, n_pml, 8.0, seed)
    return DiffProblem(shape, case["steps"], src, recs, a, a, f0=2500.0, n_pml=n_pml)


def _targets(case, seed):
    """What the receivers should have heard: smooth seeded signals."""
    rng = np.random.default_rng(seed + 9)
    t = np.arange(case["steps"])[:, None]
    return 0.01 * np.sin(2 * math.pi * t / rng.uniform(20, 60, 4) + rng.uniform(0, 6, 4))


def _amr_grid(case):
    """Cells and faces of an n^3 box whose middle fine^3 cells are split in eight
    (fine = 0: none), the outer layers absorbing."""
    n, m, dx, n_pml = case["n"], case["fine"], DX, 6
    lo = (n - m) // 2
    fine = np.zeros((n, n, n), bool)
    fine[lo:lo + m, lo:lo + m, lo:lo + m] = True
    cid = np.full((n, n, n), -1, np.int64)
    cid[~fine] = np.arange(int((~fine).sum()))
    fid = np.arange((2 * m) ** 3, dtype=np.int64).reshape(2 * m, 2 * m, 2 * m) + int((~fine).sum())
    cc = (np.argwhere(~fine) + 0.5) * dx
    fc = (np.argwhere(np.ones((2 * m,) * 3, bool)) + 0.5) * (dx / 2) + lo * dx
    centers = np.concatenate([cc, fc.reshape(-1, 3)])
    vol = np.concatenate([np.full(len(cc), dx ** 3), np.full((2 * m) ** 3, (dx / 2) ** 3)])
    ijk = np.argwhere(~fine)
    edge = np.minimum(ijk, n - 1 - ijk).min(axis=1)
    types = np.concatenate([np.where(edge < n_pml, 3, 0), np.zeros((2 * m) ** 3)]).astype(np.uint8)
    neg, pos, area, dist = [], [], [], []

    def add(a, b, s, d):
        neg.append(a.ravel())
        pos.append(b.ravel())
        area.append(np.full(a.size, s))
        dist.append(np.full(a.size, d))

    for ax in range(3):
        a, b = cid.take(range(n - 1), ax).ravel(), cid.take(range(1, n), ax).ravel()
        both = (a >= 0) & (b >= 0)
        add(a[both], b[both], dx * dx, dx)
        if m:
            add(fid.take(range(2 * m - 1), ax), fid.take(range(1, 2 * m), ax), dx * dx / 4, dx / 2)
            for side in (0, 1):   # the four fine faces of each coarse face on the level boundary
                sl = [slice(lo, lo + m)] * 3
                sl[ax] = lo - 1 if side == 0 else lo + m
                coarse = np.repeat(np.repeat(cid[tuple(sl)], 2, 0), 2, 1)
                f = fid.take(0 if side == 0 else 2 * m - 1, ax)
                add(coarse if side == 0 else f, f if side == 0 else coarse, dx * dx / 4, 0.75 * dx)
    cat = lambda x, t: np.ascontiguousarray(np.concatenate(x), dtype=t)  # noqa: E731
    return {"centers": centers, "vol": vol, "open": np.ones(len(vol)), "types": types, "neg": cat(neg, np.int32),
            "pos": cat(pos, np.int32), "area": cat(area, np.float64), "face_open": np.ones(sum(x.size for x in neg)),
            "dist": cat(dist, np.float64), "min_dx": dx / 2 if m else dx, "lo": np.zeros(3),
            "hi": np.full(3, n * dx), "n_pml": n_pml}


def _amr_pulses(g, seed):
    """Pressure pulses at seeded places: (position, value)."""
    rng = np.random.default_rng(seed + 1)
    span = float(g["hi"][0])
    return [(rng.uniform(0.25, 0.75, 3) * span, float(np.float32(rng.uniform(0.5, 2.0)))) for _ in range(4)]


# --------------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "n": case["steps"]}
    if kind == "live":
        r = _room(dict(case, n_pml=10, absorption=0.2), seed)
        f = _solver(r)
        idx, w = f.precompute_pressure_samplers(r.receiver_xyz())
        st.update(f=f, src=r.src_flat, sig=[float(s) for s in gaussian_pulse(case["steps"], 5.0)], idx=idx, w=w)
    elif kind == "room":
        r = _room(case, seed)
        f = _solver(r)
        idx, w = f.precompute_pressure_samplers(r.receiver_xyz())
        st.update(f=f, src=r.src_flat, sig=r.signal(), idx=idx, w=w,
                  p0=_moving_air((r.nx, r.ny, r.nz), seed) if case["filled"] else None)
    elif kind == "serve":
        st.update(solvers=[make_solver(r) for r in _serve_rooms(case, seed)], batch=EngineBatch())
    elif kind in ("substeps", "body"):
        b = _body(case["nx"], case["ny"], case["nz"], seed)
        drives, neck = _drives(case, b, seed)
        st.update(f=_body_solver(case, b), b=b, drives=drives, neck=[float(v) for v in neck])
    elif kind == "storage":
        st.update(room=PrecisionRoom(_storage_room(case, seed), case["mode"]))
    elif kind == "gradient":
        prob = _gradient_problem(case, seed)
        st.update(room=AdjointRoom(prob, checkpoint_every=case["every"]), targets=_targets(case, seed),
                  a=torch.tensor(prob.a, device="cuda"))
    else:
        g = _amr_grid(case)
        s = AcousticAMR(g["centers"], g["vol"], g["open"], g["types"], g["neg"], g["pos"], g["area"], g["face_open"],
                        g["dist"], C0, RHO, g["min_dx"], case["order"])
        s.set_border_condition(0, 3.0, 0.0, 0.0, g["n_pml"], g["lo"], g["hi"])
        st.update(s=s, pulses=_amr_pulses(g, seed))
    return st


def run(st):
    kind, n = st["kind"], st["n"]
    if kind == "live":
        f, out = st["f"], []
        f.reset()
        for amp in st["sig"]:
            f.add_pressure(st["src"], amp)
            f.step(1)
            out.append(f.sample_pressure_precomputed(st["idx"], st["w"]))
        return {"mics": np.stack(out), "p": f.pressure_tensor()}
    if kind == "room":
        f = st["f"]
        f.reset()
        if st["p0"] is not None:   # the start field is written through the zero-copy view
            f.pressure_tensor().copy_(st["p0"])
            torch.cuda.current_stream().synchronize()
        tr = f.run(n, st["src"], st["sig"], st["idx"], st["w"])
        return {"traces": tr, "p": f.pressure_tensor(), "v": f.velocity_tensors()}
    if kind == "serve":
        solvers, batch = st["solvers"], st["batch"]
        for f in solvers:
            f.reset()
        batch.set(solvers, [n] * len(solvers))
        batch.step(n)
        steps, status = batch.sync()
        batch.set([], [])
        return {"steps": steps, "status": status, "traces": [f.get_traces() for f in solvers],
                "p": [f.pressure_tensor() for f in solvers]}
    if kind == "substeps":
        f, b, out = st["f"], st["b"], []
        f.reset()
        for q in range(n):
            out.append(f.substep(st["drives"][q], 1.0, b["f_idx"], b["f_w"], st["neck"][q], b["s_idx"], b["s_w"]))
        return {"saddle": np.stack(out), "p": f.pressure_tensor(), "w": f.get_plate_displacement()}
    if kind == "body":
        f, b = st["f"], st["b"]
        f.reset()
        f.inject_bridge_drive(20.0 * st["drives"][n // 2], 1.0)
        f.inject_plate_force(b["f_idx"], b["f_w"], 0.2)
        f.step(n)
        return {"p": f.pressure_tensor(), "v": f.velocity_tensors(), "w": f.get_plate_displacement()}
    if kind == "storage":
        st["room"].step(n)   # the room runs on from pass to pass
        return {"p": st["room"].pressure()}
    if kind == "gradient":
        a = st["a"].detach().requires_grad_(True)
        loss = trace_loss(a, st["room"], st["targets"])
        loss.backward()
        return {"loss": loss.detach(), "grad": a.grad}
    s = st["s"]
    s.reset()
    for xyz, val in st["pulses"]:
        s.inject_pressure_nearest(xyz, val)
    s.step(n)
    return {"p": s.get_pressure(), "v": s.get_velocity()}


# ----------------------------------------------------------------------- work
def work(case):
    """Each field, coefficient and output of the pass once; the scheme's arithmetic for every step."""
    kind, n = case["kind"], case["steps"]
    if kind == "serve":
        cells = sum(r.cells for r in _serve_rooms(case, 0))
        return {"bytes": 16.0 * cells, "flops": float(CELL_FLOPS * cells * n)}
    if kind == "amr":
        g = _amr_grid(case)
        nc, nf = len(g["vol"]), g["neg"].size
        face = 24 if case["order"] == 8 else 6
        return {"bytes": 20.0 * nc + 16.0 * nf, "flops": float(n) * (face * nf + 4 * nf + 5 * nc)}
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind in ("live", "room"):
        return {"bytes": 16.0 * cells + (4.0 * cells if case.get("filled") else 0.0), "flops": float(CELL_FLOPS * cells * n)}
    if kind in ("substeps", "body"):   # three fractions and the solid mask too
        return {"bytes": (16.0 + 13.0) * cells, "flops": float((CELL_FLOPS + 3) * cells * n)}
    if kind == "storage":
        return {"bytes": 4.0 * STORAGE[case["mode"]] * cells, "flops": float(CELL_FLOPS * cells * n)}
    # gradient: one forward and one reverse sweep of every step, absorption in and gradient out
    return {"bytes": 8.0 * cells, "flops": float((CELL_FLOPS + 70) * cells * n)}


# ---------------------------------------------------------------------- exact
def _dt64(dx):
    return 0.77 * dx / (C0 * 1.732050808)


def _axis_alpha(n, n_pml, dt, lo, hi):
    a = torch.zeros(n, dtype=torch.float64, device="cuda")
    for i in range(n):
        d, s = (n_pml - i, lo) if i < n_pml else (i - (n - n_pml) + 1, hi)
        if d > 0 and n_pml > 0:
            a[i] = s * (3.45 / (dt * n_pml)) * (d / n_pml) ** 3
    return a


class _Air:
    """The staggered scheme in float64 on the GPU, walls and fractions included."""

    C1, C2 = 9.0 / 8.0, -1.0 / 24.0

    def __init__(self, shape, dx, a6, n_pml):
        self.shape, self.dt = tuple(shape), _dt64(dx)
        self.vc = self.dt / (RHO * dx)
        self.bulk = RHO * C0 * C0 * self.dt / dx
        ax = [_axis_alpha(n, n_pml, self.dt, a6[2 * q], a6[2 * q + 1]) for q, n in enumerate(shape)]
        alpha = torch.maximum(torch.maximum(ax[0][:, None, None], ax[1][None, :, None]), ax[2][None, None, :])
        self.set_damping(alpha * self.dt)
        z = lambda s: torch.zeros(s, dtype=torch.float64, device="cuda")  # noqa: E731
        self.p = z(shape)
        self.v = [z([n - (q == a) for q, n in enumerate(shape)]) for a in range(3)]
        self.fr = self.solid = None

    def set_damping(self, a):
        """a = alpha * dt per cell."""
        self.pd = 1.0 / (1.0 + a)
        self.vd = [1.0 - 0.5 * (a.narrow(q, 0, a.shape[q] - 1) + a.narrow(q, 1, a.shape[q] - 1)) for q in range(3)]

    @classmethod
    def grad(cls, p, ax):
        n = p.shape[ax]
        g = p.narrow(ax, 1, n - 1) - p.narrow(ax, 0, n - 1)
        if n >= 4:
            mid = cls.C1 * g.narrow(ax, 1, n - 3) + cls.C2 * (p.narrow(ax, 3, n - 3) - p.narrow(ax, 0, n - 3))
            g = torch.cat([g.narrow(ax, 0, 1), mid, g.narrow(ax, n - 2, 1)], dim=ax)
        return g

    @classmethod
    def div(cls, v, shape):
        d = torch.zeros(shape, dtype=torch.float64, device="cuda")
        for ax, x in enumerate(v):
            m = x.shape[ax]
            d.narrow(ax, 0, m).add_(x, alpha=cls.C1)
            d.narrow(ax, 1, m).sub_(x, alpha=cls.C1)
            if m > 1:
                d.narrow(ax, 0, m - 1).add_(x.narrow(ax, 1, m - 1), alpha=cls.C2)
                d.narrow(ax, 2, m - 1).sub_(x.narrow(ax, 0, m - 1), alpha=cls.C2)
        return d

    def step(self, plate_faces=None):
        for ax in range(3):
            self.v[ax].sub_(self.grad(self.p, ax), alpha=self.vc).mul_(self.vd[ax])
            if self.fr is not None:
                self.v[ax].masked_fill_(self.fr[ax] == 0, 0.0)
        if plate_faces is not None:
            plate_faces(self.v[2])
        v = self.v if self.fr is None else [x * f for x, f in zip(self.v, self.fr)]
        self.p = (self.p - self.bulk * self.div(v, self.shape)) * self.pd
        if self.solid is not None:
            self.p.masked_fill_(self.solid, 0.0)


def _cells(recs):
    return [torch.as_tensor([r[a] for r in recs], device="cuda") for a in range(3)]


def _run_air(air, r, n, sig):
    """Deposit, step, record; the traces (n, receivers)."""
    rec = _cells(r.receivers)
    rows = []
    for q in range(n):
        air.p[r.src] += float(sig[q])
        air.step()
        rows.append(air.p[rec[0], rec[1], rec[2]])
    return torch.stack(rows)


def _plate_biharmonic(active):
    """13-point weights with inactive neighbours replaced by the node itself, as index and weight arrays."""
    di = (0, 1, -1, 0, 0, 1, 1, -1, -1, 2, -2, 0, 0)
    dj = (0, 0, 0, 1, -1, 1, -1, 1, -1, 0, 0, 2, -2)
    wt = (20.0, -8.0, -8.0, -8.0, -8.0, 2.0, 2.0, 2.0, 2.0, 1.0, 1.0, 1.0, 1.0)
    nx, ny = active.shape
    ij = np.argwhere(active)
    idx = []
    for a, b in zip(di, dj):
        i, j = ij[:, 0] + a, ij[:, 1] + b
        ok = (i >= 0) & (i < nx) & (j >= 0) & (j < ny)
        ok &= active[np.clip(i, 0, nx - 1), np.clip(j, 0, ny - 1)]
        idx.append(np.where(ok, j + ny * i, ij[:, 1] + ny * ij[:, 0]))
    return torch.as_tensor(np.stack(idx), device="cuda"), torch.tensor(wt, dtype=torch.float64, device="cuda")[:, None]


def _exact_body(case, seed, forces):
    """Plate, walls and air in float64; forces(q) = {node: force} before step q.  Returns air, w, saddle rows."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    b = _body(nx, ny, nz, seed)
    air = _Air((nx, ny, nz), BODY_DX, (1.0,) * 6, 6)
    air.fr = [torch.as_tensor(x, device="cuda").double() for x in b["fr"]]
    air.solid = torch.as_tensor(b["ct"] > 0, device="cuda")
    dt, piz, act = air.dt, b["piz"], b["active"]
    i, j = (torch.as_tensor(x, device="cuda") for x in np.nonzero(act))
    node = j + ny * i
    nb, wt = _plate_biharmonic(act)
    below_open = torch.as_tensor(b["ct"][:, :, piz - 1][act] == 0, device="cuda")
    above_open = torch.as_tensor(b["ct"][:, :, piz + 1][act] == 0, device="cuda")
    m, dd = 7.0, 0.45
    ka, kb = dt * dt / m, dd * dt * dt / (m * BODY_DX ** 4)
    vd, bk = 1.0 - 2.0 * dt, 1e-5 / dt * kb
    w = torch.zeros(nx * ny, dtype=torch.float64, device="cuda")
    wp = w.clone()
    s_idx = torch.as_tensor(b["s_idx"], device="cuda").long().reshape(-1, 4)
    rows = []
    for q in range(case["steps"]):
        ext = torch.zeros_like(w)
        for idx, val in forces(b, q):
            ext.index_add_(0, torch.as_tensor(idx, device="cuda").long(),
                           torch.as_tensor(np.asarray(val, np.float64) / BODY_DX ** 2, device="cuda"))
        bh, bhp = (wt * w[nb]).sum(0), (wt * wp[nb]).sum(0)
        new = w[node] + vd * (w[node] - wp[node]) - kb * bh - bk * (bh - bhp)
        new = new + ka * (air.p[i, j, piz - 1] - air.p[i, j, piz + 1] + ext[node])
        wn = w.clone()
        wn[node] = new
        w, wp = wn, w
        vel = (w[node] - wp[node]) / dt

        def faces(vz):
            vz[i[below_open], j[below_open], piz - 1] = vel[below_open]
            vz[i[above_open], j[above_open], piz] = vel[above_open]

        air.step(faces)
        rows.append((w[s_idx] * 0.25).sum(1))
    return air, w.reshape(nx, ny), torch.stack(rows)


def _exact_gradient(case, seed):
    from torch.utils.checkpoint import checkpoint
    prob = _gradient_problem(case, seed)
    a = torch.tensor(prob.a, device="cuda").double().requires_grad_(True)
    shape, dt = prob.shape, _dt64(prob.dx)
    vc, bulk = dt / (RHO * prob.dx), RHO * C0 * C0 * dt / prob.dx
    sig = np.asarray(prob.signal(), np.float64)
    rec = _cells(prob.receivers)
    src = torch.zeros(shape, dtype=torch.float64, device="cuda")
    src[prob.src] = 1.0
    pad = [(0, 0, 0, 0, 2, 2), (0, 0, 2, 2, 0, 0), (2, 2, 0, 0, 0, 0)]

    def steps(n0, n1, a, p, vx, vy, vz):
        pd = 1.0 / (1.0 + a)
        v, rows = [vx, vy, vz], []
        for q in range(n0, n1):
            p = p + float(sig[q]) * src
            d = 0
            for ax in range(3):
                n = shape[ax]
                vd = 1.0 - 0.5 * (a.narrow(ax, 0, n - 1) + a.narrow(ax, 1, n - 1))
                v[ax] = (v[ax] - vc * _Air.grad(p, ax)) * vd
                x = torch.nn.functional.pad(v[ax], pad[ax])
                d = d + _Air.C1 * (x.narrow(ax, 2, n) - x.narrow(ax, 1, n)) \
                    + _Air.C2 * (x.narrow(ax, 3, n) - x.narrow(ax, 0, n))
            p = (p - bulk * d) * pd
            rows.append(p[rec[0], rec[1], rec[2]])
        return (p, *v, torch.stack(rows))

    st = [torch.zeros(shape, dtype=torch.float64, device="cuda")]
    st += [torch.zeros([n - (q == ax) for q, n in enumerate(shape)], dtype=torch.float64, device="cuda") for ax in range(3)]
    out = []
    for n0 in range(0, case["steps"], 16):
        *st, rows = checkpoint(steps, n0, min(n0 + 16, case["steps"]), a, *st, use_reentrant=False)
        out.append(rows)
    loss = ((torch.cat(out) - torch.as_tensor(_targets(case, seed), device="cuda")) ** 2).sum()
    loss.backward()
    return {"loss": loss.detach(), "grad": a.grad}


def _order8_weights():
    """Weights (unit spacing) of the first to fourth pair of cells beside a face,
    by the recurrence the reference's order-8 stencil is defined with."""
    x = np.arange(8) - 3.5
    c0, c1, before = np.zeros(8), np.zeros(8), 1.0
    c0[0] = 1.0
    for a in range(1, 8):
        here = 1.0
        for b in range(a):
            d = x[a] - x[b]
            here *= d
            if b == a - 1:
                c1[a] = before / here * (c0[b] - x[a] * c1[b])
                c0[a] = before / here * -x[a] * c0[b]
            c1[b] = (x[a] * c1[b] - c0[b]) / d
            c0[b] = x[a] * c0[b] / d
        before = here
    return [float(c1[4 + k]) for k in range(4)]


def _exact_amr(case, seed):
    g = _amr_grid(case)
    dev = lambda x: torch.as_tensor(x, device="cuda")  # noqa: E731
    nc = len(g["vol"])
    order = case["order"]
    dt = (0.10 if order == 8 else 0.77) * g["min_dx"] / (C0 * math.sqrt(3.0))
    neg, pos = dev(g["neg"]).long(), dev(g["pos"]).long()
    flux, vol = dev(g["area"]), dev(g["vol"])
    # absorbing border: alpha from the depth inside the layer, exponential damping
    c = dev(g["centers"])
    d = torch.minimum(c - dev(g["lo"]), dev(g["hi"]) - c).min(dim=1).values.clamp(min=0.0)
    depth = g["n_pml"] * dt * C0 * math.sqrt(3.0) / 0.77
    alpha = 3.45 / (dt * g["n_pml"]) * (1.0 - d / depth).clamp(0.0, 1.0) ** 3
    alpha = torch.where(dev(g["types"]) == 3, alpha, torch.zeros_like(alpha))
    s = alpha * dt
    pdamp = torch.exp(-s)
    psrc = torch.where(s < 1e-6, 1.0 - 0.5 * s, (1.0 - torch.exp(-s)) / s.clamp(min=1e-300))
    vdamp = torch.exp(-(alpha[neg] + alpha[pos]) * dt)
    p = torch.zeros(nc, dtype=torch.float64, device="cuda")
    v = torch.zeros(neg.numel(), dtype=torch.float64, device="cuda")
    for xyz, val in _amr_pulses(g, seed):
        p[int(((c - dev(xyz)) ** 2).sum(1).argmin())] += val
    bulk, n = RHO * C0 * C0 * dt, case["n"]
    wide = _order8_weights()
    for _ in range(case["steps"]):
        if order == 8:   # one level: eight points where four cells lie on each side, else two
            q, gr = p.reshape(n, n, n), []
            for ax in range(3):
                f = q.narrow(ax, 1, n - 1) - q.narrow(ax, 0, n - 1)
                m = n - 7
                mid = sum(wide[k] * (q.narrow(ax, 4 + k, m) - q.narrow(ax, 3 - k, m)) for k in range(4))
                gr.append(torch.cat([f.narrow(ax, 0, 3), mid, f.narrow(ax, n - 4, 3)], dim=ax).ravel() / DX)
            gr = torch.cat(gr)
        else:
            gr = (p[pos] - p[neg]) / dev(g["dist"])
        v = (v - dt / RHO * gr) * vdamp
        dv = torch.zeros_like(p).index_add_(0, neg, flux * v).index_add_(0, pos, -flux * v)
        p = p * pdamp - bulk * dv / vol * psrc
    return {"p": p, "v": v}


def exact(case, seed):
    kind, n = case["kind"], case["steps"]
    if kind == "live":
        r = _room(dict(case, n_pml=10, absorption=0.2), seed)
        air = _Air((r.nx, r.ny, r.nz), DX, r.absorption, 10)
        tr = _run_air(air, r, n, gaussian_pulse(n, 5.0))
        return {"mics": tr, "p": air.p}
    if kind == "room":
        r = _room(case, seed)
        air = _Air((r.nx, r.ny, r.nz), DX, r.absorption, r.n_pml)
        if case["filled"]:
            air.p += _moving_air((r.nx, r.ny, r.nz), seed)
        tr = _run_air(air, r, n, r.signal())
        return {"traces": tr, "p": air.p, "v": tuple(air.v)}
    if kind == "serve":
        tr, ps = [], []
        for r in _serve_rooms(case, seed):
            air = _Air((r.nx, r.ny, r.nz), DX, r.absorption, r.n_pml)
            tr.append(_run_air(air, r, n, r.signal()))
            ps.append(air.p)
        return {"steps": None, "status": None, "traces": tr, "p": ps}
    if kind in ("substeps", "body"):
        drives, neck = _drives(case, _body(case["nx"], case["ny"], case["nz"], seed), seed)

        def forces(b, q):
            if kind == "substeps":
                return [(b["b_node"], drives[q].astype(np.float64)), (b["f_idx"], float(neck[q]) * b["f_w"].astype(np.float64))]
            if q > 0:
                return []
            return [(b["b_node"], (20.0 * drives[n // 2]).astype(np.float32).astype(np.float64)),
                    (b["f_idx"], float(np.float32(0.2)) * b["f_w"].astype(np.float64))]

        air, w, rows = _exact_body(case, seed, forces)
        if kind == "substeps":
            return {"saddle": rows, "p": air.p, "w": w}
        return {"p": air.p, "v": tuple(air.v), "w": w}
    if kind == "storage":   # the first pass
        r = _storage_room(case, seed)
        air = _Air((r.nx, r.ny, r.nz), DX, r.absorption, r.n_pml)
        _run_air(air, r, n, r.signal())
        return {"p": air.p}
    if kind == "gradient":
        return _exact_gradient(case, seed)
    return _exact_amr(case, seed)


if __name__ == "__main__":
    for c in listed():
        w = work(c)
        print(f"{c['name']:16s} {w['bytes'] / 1e6:10.1f} MB {w['flops'] / 1e9:10.1f} Gflop")
