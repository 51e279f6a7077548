"""The multigrid-preconditioned pressure solve at the sizes where its tiling can go wrong, against the oracle's CG on the
same velocities and marks: extents one below, at and one above the 8-cell tiles and the halvings of the levels, grids a
cell or two thin, unequal spacings, and fluid that is a block, a block with spray (tiles of a few cells, which the
solver takes out of its V-cycle) and a sponge of single cells and holes.

Tolerance: both solves stop on |b - A p| <= t |b|, so |p - p'| <= (t + t') cond(A) |p|.  With the extents used (at most 72
cells, spacings within a factor 2) cond(A) <= 12 * 4 * (4 * 72^2 / pi^2) = 1.01e5, which with t = 1e-10 and the
oracle's 1e-12 gives 1.03e-5.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")


def fluid_cells(n, kind, rng):
    i, j, k = np.meshgrid(*[np.arange(m) for m in n], indexing="ij")
    block = (i < max(1, int(0.5 * n[0]))) & (j < max(1, int(0.7 * n[1])))
    if kind == "block":
        return block
    if kind == "spray":
        return block | (rng.random(n) < 0.004)
    return rng.random(n) < 0.6


@pytest.mark.parametrize("kind", ["block", "spray", "sponge"])
@pytest.mark.parametrize("n,h", [((9, 8, 8), 1.0), ((12, 12, 12), 1.0), ((17, 9, 8), 1.0), ((8, 8, 65), 1.0),
                                 ((2, 2, 40), 1.0), ((31, 33, 30), 1.0), ((40, 24, 56), 1.0), ((72, 70, 66), 1.0),
                                 ((24, 20, 16), (1.0, 1.5, 2.0))])
def test_multigrid_solve_matches_oracle(n, h, kind):
    rng = np.random.default_rng(sum(n))
    h = np.ones(3) * h / 64.0
    size = tuple(float(h[a] * n[a]) for a in range(3))
    cells = np.argwhere(fluid_cells(n, kind, rng))
    # one particle at a cell's centre marks that cell; with unequal spacings its neighbours too
    pos = ((cells + 0.5) * h).astype(np.float32)
    vel = rng.standard_normal(pos.shape).astype(np.float32)
    g = fe.Scene(n, solver=fe.PIC, size=size, max_cfl=1.0, cg_rel_tol=1e-10, cg_max_it=2000, max_refine=40,
                 pressure_solver=fe.MGPCG)
    g.set_particles(pos, vel)
    dt = 1 / 240
    g.run_stages(dt, fe.STAGE_SORT, fe.STAGE_PRE)
    u, v, w, _, marks = g.grid()
    assert marks.sum() >= len(cells)
    g.run_stages(dt, fe.STAGE_PRESSURE, fe.STAGE_PRESSURE)
    p = g.grid()[3]
    assert g.tuning()["multigrid"] == 1
    U, V, W = (a.astype(np.float64) for a in (u, v, w))
    expected = np.zeros_like(p)
    _, res = oracle.project(n, h, marks, U, V, W, expected, rel_tol=1e-12, max_it=20000)
    assert res <= 1e-12
    assert np.linalg.norm(p - expected) <= 1.03e-5 * np.linalg.norm(expected)
    g.close()


def test_scenes_of_different_block_sizes():
    """A scene of smaller solver blocks prepared after one of larger blocks, both stepped afterwards."""
    scenes = []
    for threads in (1024, 512, 256):
        g = fe.Scene((32, 32, 32), solver=fe.FLIP, max_cfl=1.0)
        g.set_tuning(multigrid=1, cg_block_threads=threads)
        pos, _ = fe.seed_regions([dict(kind=0, lo=(0, 0, 0), hi=(0.4, 0.6, 1.0))], (32, 32, 32), (0, 0, 0), (1, 1, 1), 3)
        g.set_particles(pos, np.zeros_like(pos))
        scenes.append(g)
    for g in scenes:
        assert all(s["converged"] == 1 for s in g.step(1 / 240, 2))
        g.close()
