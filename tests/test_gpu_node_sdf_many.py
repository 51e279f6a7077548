"""The fluid's band SDF gathered from the particles' cells, which scenes of many particles take, bit for bit against the oracle:
crowded cells (around the 32 particles a thread tests, and some thousands) next to empty ones, cell corners, lone particles,
tile edges, exact and inexact node positions, an origin away from zero; from cells grouped for the surface and from those of
the sort; and the particle counts from which either is taken."""
import ctypes

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")
from fluide_engine_b200._abi import check  # noqa: E402

DT = 1 / 240
GRIDS = [((40, 56, 48), 1 / 64, (0, 0, 0)), ((47, 41, 58), 1 / 60, (0, 0, 0)), ((50, 48, 44), 1 / 50, (-0.5, 0.25, 1.0))]
KINDS = ["block", "spray", "corners", "crowded", "cap"]


def particles(n, h, origin, kind, count, rng):
    """At least `count` particles in any order."""
    n = np.asarray(n)
    if kind == "spray":
        pos = np.repeat(rng.uniform(0, 1, (4000, 3)) * n * h, count // 4000 + 1, axis=0)
    elif kind == "corners":  # exactly on cell corners
        pos = np.repeat(rng.integers(0, n + 1, (9000, 3)) * h, count // 9000 + 1, axis=0)
    elif kind == "crowded":
        at = (rng.integers(0, n, (count // 60, 3)) + 0.5) * h
        pos = np.repeat(at, rng.integers(20, 140, len(at)), axis=0)
        pos = pos + rng.uniform(-0.6, 0.6, pos.shape) * h
    elif kind == "cap":
        cells = rng.permutation(np.argwhere(np.ones(n, bool)))[:count // 25]
        reps = rng.choice([1, 30, 31, 32, 33, 34], len(cells))
        reps[:6] = [63, 64, 65, 1000, 1025, 3000]
        pos = (np.repeat(cells, reps, axis=0) + rng.uniform(0, 1, (reps.sum(), 3))) * h
    else:
        per = 3 if count > 1 << 19 else 2
        m = np.stack(np.meshgrid(*[np.arange(per * k) for k in n], indexing="ij"), -1).reshape(-1, 3)
        pos = (m + rng.uniform(0, 1, m.shape)) * h / per
        pos = pos[(pos[:, 0] < 0.61 * n[0] * h) & (pos[:, 1] < 0.83 * n[1] * h)]
    assert len(pos) >= count
    return (np.clip(pos, 0, n * h) + np.asarray(origin))[rng.permutation(len(pos))].astype(np.float32)


def expected(n, h, origin, pos, **kw):
    o = oracle.OracleSim(n, oracle.FLIP, origin=origin, size=tuple(h * k for k in n), **kw)
    o.set_particles(pos.astype(np.float64))
    o.stage("sdf")
    return o


def scene(n, h, origin, pos, **kw):
    g = fe.Scene(n, solver=fe.FLIP, origin=origin, size=tuple(h * k for k in n), max_cfl=1.0, **kw)
    g.set_particles(pos, np.zeros_like(pos))
    return g


def launches(f):
    before = fe.kernel_launch_count()
    f()
    return fe.kernel_launch_count() - before


def surface_launches(g):
    a, b = ctypes.c_uint64(), ctypes.c_uint64()
    return launches(lambda: check(fe.lib().fe_scene_build_surface(g.handle, ctypes.byref(a), ctypes.byref(b))))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,h,origin", GRIDS)
def test_surface_of_unsorted_particles(n, h, origin, kind):
    pos = particles(n, h, origin, kind, 1 << 20, np.random.default_rng(n[0] + len(kind)))
    g = scene(n, h, origin, pos)
    o = expected(n, h, origin, pos)
    d = [h * k / k for k in n]
    mesh = oracle.build_surface(o.sdf(), n, [origin[a] + d[a] / 2.0 for a in range(3)], d)
    for a, b in zip(g.surface(), mesh):
        assert np.array_equal(a, b)
    g.close()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n,h,origin", GRIDS)
def test_viscous_faces_of_sorted_particles(n, h, origin, kind):
    pos = particles(n, h, origin, kind, 1 << 18, np.random.default_rng(3 + n[0] + len(kind)))
    g = scene(n, h, origin, pos, viscosity=0.01)
    g.run_stages(DT, fe.STAGE_SORT, fe.STAGE_PRE)
    g.run_stages(DT, fe.STAGE_DIFFUSE, fe.STAGE_DIFFUSE)
    o = expected(n, h, origin, pos, viscosity=0.01)
    o.stage("p2g")
    o.stage("diffusion", DT)
    for a, b in zip(g.diffusion()[1], o.diffusion_markers()):
        assert np.array_equal(a, b)
    g.close()


def test_particle_counts():
    """Grouped for the surface from 2^20 particles on (sort's passes and one gather for two scatter passes), from the sort's cells
    from 2^18 on."""
    n, h, origin = GRIDS[0]
    pos = particles(n, h, origin, "block", 1 << 20, np.random.default_rng(7))
    few, many = scene(n, h, origin, pos[:(1 << 20) - 1]), scene(n, h, origin, pos[:1 << 20])
    assert surface_launches(many) == surface_launches(few) + 4
    few.close()
    many.close()
    diffuse = []
    for count in ((1 << 18) - 1, 1 << 18):
        g = scene(n, h, origin, pos[:count], viscosity=0.01)
        g.run_stages(DT, fe.STAGE_SORT, fe.STAGE_PRE)
        diffuse.append(launches(lambda: g.run_stages(DT, fe.STAGE_DIFFUSE, fe.STAGE_DIFFUSE)))
        g.close()
    assert diffuse[1] == diffuse[0] - 1
