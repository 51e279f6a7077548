"""The pressure of a tank full of fluid: without an AIR cell the system determines it up to a constant, and CG from a given
start keeps the start's mean.  Against the oracle's CG from the same pressure, for every solver choice, alone and in a batch.

Tolerance: both solves stop on |b - A p| <= t |b|, so apart from the constant |p - p'| <= (t + t') cond(A) |p|, with cond(A) <=
12 / (4 sin^2(pi / 2 n)) <= 3 n^2 for n cells along the longest axis: t = 1e-10, t' = 1e-12 and n <= 40 give 4.9e-7.  The
constant: the FP32 corrections of up to 1e-2 per cell are summed to zero up to their rounding, 6e-8 |p| each, of at most 40
refinements: 2.4e-6 in all."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")
from fluide_engine_b200._abi import check, ptr  # noqa: E402

GRIDS = [(8, 16, 8), (12, 12, 12), (20, 17, 23), (32, 32, 32), (40, 33, 9)]
H = 1.0 / 64
DT = 1 / 240


def tank(n, pressure_solver, rng):
    cells = np.argwhere(np.ones(n, bool))
    pos = ((cells + 0.5) * H).astype(np.float32)
    g = fe.Scene(n, solver=fe.PIC, size=tuple(H * k for k in n), max_cfl=1.0, cg_rel_tol=1e-10, cg_max_it=4000, max_refine=40,
                 pressure_solver=pressure_solver)
    g.set_particles(pos, rng.standard_normal(pos.shape).astype(np.float32))
    return g


def close(p, n, marks, u, v, w, start):
    assert marks.min() == marks.max() == 1
    e = np.ascontiguousarray(start, dtype=np.float64).copy()
    _, res = oracle.project(n, (H,) * 3, marks, *(a.astype(np.float64) for a in (u, v, w)), e, rel_tol=1e-12, max_it=20000)
    assert res <= 1e-12
    assert np.linalg.norm(p - e) <= 2.9e-6 * np.linalg.norm(e)


@pytest.mark.parametrize("start", ["zero", "warm"])
@pytest.mark.parametrize("solver", [fe.AUTO, fe.MGPCG, fe.CG])
@pytest.mark.parametrize("n", GRIDS)
def test_mean_pressure_is_kept(n, solver, start):
    rng = np.random.default_rng(sum(n))
    g = tank(n, solver, rng)
    p0 = np.zeros((n[2], n[1], n[0]))
    if start == "warm":
        p0 = 1e-3 * (2.0 + rng.standard_normal(p0.shape))
    check(fe.lib().fe_scene_set_pressure(g.handle, ptr(p0)))
    g.run_stages(DT, fe.STAGE_SORT, fe.STAGE_PRE)
    u, v, w, _, marks = g.grid()
    g.run_stages(DT, fe.STAGE_PRESSURE, fe.STAGE_PRESSURE)
    close(g.grid()[3], n, marks, u, v, w, p0)
    g.close()


def test_mean_pressure_is_kept_in_a_batch():
    rng = np.random.default_rng(1)
    scenes = [tank(n, fe.AUTO, rng) for n in GRIDS]
    grids = []
    for g in scenes:
        snap = g.checkpoint()
        g.run_stages(DT, fe.STAGE_SORT, fe.STAGE_PRE)
        grids.append(g.grid())
        g.restore(snap)
    batch = fe.Batch(scenes)
    batch.step(DT, 1)
    for n, g, (u, v, w, _, marks) in zip(GRIDS, scenes, grids):
        close(g.grid()[3], n, marks, u, v, w, np.zeros((n[2], n[1], n[0])))
    batch.close()
