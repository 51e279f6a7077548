"""Cell marks where the two-pass marking can go wrong, bit for bit against the oracle: particles piled into corners (out of
reach of their own cell's centre), crowded cells next to empty ones, tile edges, lone particles, grids with inexact
cell-centre samples, unequal spacings (marked particle by particle); and marks of particles that moved since the sort."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")


def particles(n, size, kind, rng):
    size = np.asarray(size)
    h = size / np.asarray(n)
    if kind == "spray":
        pos = rng.uniform(0, 1, (60, 3)) * size
    elif kind == "corners":  # exactly on cell corners and on the domain's corners, many per cell
        at = rng.integers(0, np.asarray(n) + 1, (40, 3)) * h
        pos = np.repeat(np.concatenate([at, np.array([[0, 0, 0], size])]), 45, axis=0)
    elif kind == "crowded":
        at = (rng.integers(0, n, (12, 3)) + 0.5) * h
        pos = np.repeat(at, rng.integers(20, 120, 12), axis=0)
        pos = pos + rng.uniform(-0.6, 0.6, pos.shape) * h
    else:
        m = np.stack(np.meshgrid(*[np.arange(2 * k) for k in n], indexing="ij"), -1).reshape(-1, 3)
        pos = (m + rng.uniform(0, 1, m.shape)) * h / 2
        pos = pos[(pos[:, 0] < 0.43 * size[0]) & (pos[:, 1] < 0.71 * size[1])]
    return np.clip(pos, 0, size).astype(np.float32)


@pytest.mark.parametrize("kind", ["block", "spray", "corners", "crowded"])
@pytest.mark.parametrize("n,size", [((16, 16, 16), (1, 1, 1)), ((9, 17, 7), (9 / 16, 17 / 16, 7 / 16)),
                                    ((24, 8, 25), (0.96, 0.32, 1.0)), ((12, 20, 10), (1, 1, 1))])
def test_marks_match_oracle(n, size, kind):
    rng = np.random.default_rng(n[0] + len(kind))
    pos = particles(n, size, kind, rng)
    g = fe.Scene(n, solver=fe.FLIP, size=size, max_cfl=1.0)
    g.set_particles(pos, np.zeros_like(pos))
    g.run_stages(1 / 240, fe.STAGE_SORT, fe.STAGE_MARK)
    o = oracle.OracleSim(n, oracle.FLIP, size=size)
    o.set_particles(pos.astype(np.float64))
    o.stage("sdf")
    o.stage("markers")
    assert np.array_equal(g.grid()[4], o.marks())
    g.close()


def test_marks_of_moved_particles():
    """The marking stage alone after a move (the cell starts are the sort's, the positions are not) and on a batch."""
    n = (24, 24, 24)
    rng = np.random.default_rng(4)
    pos = particles(n, (1, 1, 1), "block", rng)
    vel = (rng.standard_normal(pos.shape) * 4).astype(np.float32)
    a = fe.Scene(n, solver=fe.FLIP, max_cfl=1.0)
    a.set_particles(pos, vel)
    a.step(1 / 60, 2)
    moved = a.particles()[0]
    a.run_stages(1 / 60, fe.STAGE_MARK, fe.STAGE_MARK)
    b = fe.Scene(n, solver=fe.FLIP, max_cfl=1.0)
    b.set_particles(moved, np.zeros_like(moved))
    b.run_stages(1 / 60, fe.STAGE_SORT, fe.STAGE_MARK)
    assert np.array_equal(a.grid()[4], b.grid()[4])
    a.close()
    b.close()


def test_flat_batch_marks_both_ways():
    """One flat launch over grids marked cell by cell and particle by particle."""
    scenes, alone = [], []
    for k, (n, size) in enumerate([((16, 16, 16), (1, 1, 1)), ((12, 20, 10), (1, 1, 1)), ((24, 8, 25), (0.96, 0.32, 1.0))]):
        pos = particles(n, size, "block", np.random.default_rng(k))
        for group in (scenes, alone):
            s = fe.Scene(n, solver=fe.FLIP, size=size, max_cfl=1.0)
            s.set_particles(pos, np.zeros_like(pos))
            group.append(s)
    batch = fe.Batch(scenes)
    batch.set_flat(-1)
    batch.step(1 / 240, 1)
    for s, t in zip(scenes, alone):
        t.step(1 / 240, 1)
        assert np.array_equal(s.grid()[4], t.grid()[4])
    batch.close()
