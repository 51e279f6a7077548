"""The marking in two passes (each particle's own cell, then the cells next to an unmarked one), which scenes of many sorted
particles take, bit for bit against the oracle: particles piled into corners (out of reach of their own cell's centre),
crowded cells next to empty ones, lone particles, tile edges, a lattice (particles at a node's radius), exact and inexact
cell-centre samples, an origin away from zero; marks of particles that moved since the sort; and the particle counts from
which it is taken."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")

DT = 1 / 240
EXACT = ((40, 56, 48), 1 / 64, (0, 0, 0))
GRIDS = [EXACT, ((47, 41, 58), 1 / 60, (0, 0, 0)), ((50, 48, 44), 1 / 50, (-0.5, 0.25, 1.0))]
KINDS = ["block", "spray", "corners", "crowded", "cap", "lattice"]


def particles(n, h, origin, kind, count, rng):
    """At least `count` particles, or exactly so many ("exactly")."""
    n = np.asarray(n)
    if kind == "spray":
        pos = np.repeat(rng.uniform(0, 1, (8000, 3)) * n * h, count // 8000 + 1, axis=0)
    elif kind == "corners":  # exactly on cell corners
        pos = np.repeat(rng.integers(0, n + 1, (20000, 3)) * h, count // 20000 + 1, axis=0)
    elif kind == "crowded":
        at = (rng.integers(0, n, (count // 60, 3)) + 0.5) * h
        pos = np.repeat(at, rng.integers(20, 140, len(at)), axis=0)
        pos = pos + rng.uniform(-0.6, 0.6, pos.shape) * h
    elif kind == "cap":  # one cell each, around the 64 particles that 8 lanes test, and some hundreds and thousands
        cells = rng.permutation(np.argwhere(np.ones(n, bool)))[:count // 62]
        reps = rng.choice([61, 62, 63, 64, 65, 66, 67], len(cells))
        reps[:7] = [255, 256, 257, 1023, 1025, 2049, 3000]
        pos = (np.repeat(cells, reps, axis=0) + rng.uniform(0, 1, (reps.sum(), 3))) * h
    else:  # a block of fluid, 3^3 a cell; on a lattice of 5 x 5 x 1 some are 0.6 h away from a node along x and y: its radius
        per = np.array([3, 3, 3] if kind != "lattice" else [5, 5, 1])
        m = np.stack(np.meshgrid(*[np.arange(p * k) for p, k in zip(per, n)], indexing="ij"), -1).reshape(-1, 3)
        pos = (m + (0.5 if kind == "lattice" else rng.uniform(0, 1, m.shape))) * h / per
        pos = pos[(pos[:, 0] < 0.61 * n[0] * h) & (pos[:, 1] < 0.83 * n[1] * h)]
    pos = (np.clip(pos, 0, n * h) + np.asarray(origin))[rng.permutation(len(pos))].astype(np.float32)
    if kind == "exactly":
        return np.concatenate([pos, pos[:max(0, count - len(pos))]])[:count]
    assert len(pos) >= count
    return pos


def scene(n, h, origin, pos, vel=None):
    g = fe.Scene(n, solver=fe.FLIP, origin=origin, size=tuple(h * k for k in n), max_cfl=1.0)
    g.set_particles(pos, np.zeros_like(pos) if vel is None else vel)
    return g


def mark_launches(g):
    before = fe.kernel_launch_count()
    g.run_stages(DT, fe.STAGE_MARK, fe.STAGE_MARK)
    return fe.kernel_launch_count() - before


def marks(n, h, origin, pos):
    o = oracle.OracleSim(n, oracle.FLIP, origin=origin, size=tuple(h * k for k in n))
    o.set_particles(pos.astype(np.float64))
    o.stage("sdf")
    o.stage("markers")
    return o.marks()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,h,origin", GRIDS)
def test_marks_match_oracle(n, h, origin, kind):
    pos = particles(n, h, origin, kind, 1 << 20, np.random.default_rng(n[0] + len(kind)))
    g = scene(n, h, origin, pos)
    g.run_stages(DT, fe.STAGE_SORT, fe.STAGE_PRE)
    assert mark_launches(g) == (2 if (n, h, origin) == EXACT else 3)  # two passes, and the exact test of inexact samples
    assert np.array_equal(g.grid()[4], marks(n, h, origin, pos))
    g.close()


@pytest.mark.parametrize("n,h,origin", GRIDS)
def test_marks_of_moved_particles(n, h, origin):
    """After a move the cell starts are no longer the positions': one pass over the particles, until the next sort."""
    rng = np.random.default_rng(4)
    pos = particles(n, h, origin, "block", 1 << 20, rng)
    g = scene(n, h, origin, pos, (rng.standard_normal(pos.shape) * 4).astype(np.float32))
    g.step(DT, 2, stats=False)
    exact = (n, h, origin) == EXACT
    assert mark_launches(g) == (1 if exact else 2)
    moved = g.particles()[0]
    expected = marks(n, h, origin, moved)
    assert np.array_equal(g.grid()[4], expected)
    g.run_stages(DT, fe.STAGE_SORT, fe.STAGE_PRE)
    assert mark_launches(g) == (2 if exact else 3)
    assert np.array_equal(g.grid()[4], expected)
    g.close()


@pytest.mark.parametrize("grid,count,passes", [(0, (1 << 20) - 1, 1), (0, 1 << 20, 2), (0, 1 << 19, 1), (1, (1 << 19) - 1, 1),
                                               (1, 1 << 19, 2)])
def test_particle_counts(grid, count, passes):
    """Two passes from 2^20 particles on, and from 2^19 on where cell-centre samples are inexact."""
    n, h, origin = GRIDS[grid]
    pos = particles(n, h, origin, "exactly", count, np.random.default_rng(7))
    assert len(pos) == count
    g = scene(n, h, origin, pos)
    g.run_stages(DT, fe.STAGE_SORT, fe.STAGE_PRE)
    assert mark_launches(g) == passes + (1 if grid else 0)
    assert np.array_equal(g.grid()[4], marks(n, h, origin, pos))
    g.close()
