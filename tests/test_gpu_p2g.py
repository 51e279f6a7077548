"""Particle-to-grid sums where the block's division of the work can go wrong, against the oracle: quarter tiles around the
count below which particles go straight to the grid, cells around the count a thread sums by itself, cells of very unequal
counts, the first and last cells of every axis (the clamps of either cell or face counts), particles exactly on faces, grids
with ragged tiles, two cells an axis, and domain origins away from zero.  Cells are powers of two, so the faces a particle
touches are the same in 32 and 64 bits; the sums differ by the rounding of up to a few hundred terms (1e-5 relative)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")


def particles(n, h, kind, rng):
    n = np.asarray(n)
    if kind == "few":      # 31, 32, 33 and 34 particles in the first two layers of a tile, others nearly empty
        count = 31 + int(rng.integers(0, 4))
        pos = rng.uniform(0, 1, (count, 3)) * np.minimum(n, [8, 8, 2]) * h
        pos = np.concatenate([pos, rng.uniform(0, 1, (7, 3)) * n * h])
    elif kind == "crowded":  # 31 .. 34 and some hundred particles a cell
        at = rng.integers(0, n, (9, 3))
        reps = np.array([31, 32, 33, 34, 63, 64, 65, 150, 300])
        pos = (np.repeat(at, reps, axis=0) + rng.uniform(0, 1, (reps.sum(), 3))) * h
    elif kind == "walls":
        pos = rng.uniform(0, 1, (4000, 3)) * n * h
        for a in range(3):
            low, high = rng.integers(0, 4000, 500), rng.integers(0, 4000, 500)
            pos[low, a] = rng.choice([0.0, 0.25, 0.5, 1.0], 500) * h
            pos[high, a] = n[a] * h - rng.choice([0.0, 0.25, 0.5, 1.0], 500) * h
    else:
        pos = rng.uniform(0, 1, (int(8 * n.prod()), 3)) * n * h
    return np.clip(pos, 0, n * h).astype(np.float32)


@pytest.mark.parametrize("solver", [fe.PIC, fe.FLIP, fe.APIC])
@pytest.mark.parametrize("kind", ["few", "crowded", "walls", "full"])
@pytest.mark.parametrize("n,origin", [((16, 8, 8), (0, 0, 0)), ((9, 17, 7), (0, 0, 0)), ((2, 3, 2), (0, 0, 0)),
                                      ((10, 9, 11), (-0.25, 0.125, 0.5))])
def test_sums_match_oracle(n, origin, kind, solver):
    h = 1.0 / 16
    rng = np.random.default_rng(100 * n[0] + 10 * len(kind) + n[1])
    pos = particles(n, h, kind, rng) + np.asarray(origin, dtype=np.float32)
    vel = rng.standard_normal(pos.shape).astype(np.float32)
    C = rng.standard_normal((len(pos), 3, 3)).astype(np.float32) if solver == fe.APIC else None
    size = tuple(h * k for k in n)
    g = fe.Scene(n, solver=solver, origin=origin, size=size, max_cfl=1.0)
    g.set_particles(pos, vel, C)
    g.run_stages(1 / 240, fe.STAGE_SORT, fe.STAGE_P2G)
    o = oracle.OracleSim(n, solver, origin=origin, size=size)
    o.set_particles(pos.astype(np.float64), vel.astype(np.float64), None if C is None else C.astype(np.float64))
    o.stage("p2g")
    for a, b in zip(g.face_markers(), o.face_markers()):
        assert np.array_equal(a, b)
    for a, b in zip(g.grid()[:3], o.grid()):
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
    g.close()
