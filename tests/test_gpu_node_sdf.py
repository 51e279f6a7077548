"""The fluid's band SDF per node, gathered from the particles' cells, where that can go wrong, bit for bit against the oracle:
particles in cell corners (no node's own cell decides), crowded cells (spread over a warp) next to empty ones, lone particles
(every node of their surroundings is searched), tile edges, inexact node positions, an origin away from zero, and spacings so
unequal that the band is wider than the gather's reach (the scatter over particles)."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")

GRIDS = [((16, 16, 16), (1, 1, 1), (0, 0, 0)), ((34, 6, 66), (34 / 32, 6 / 32, 66 / 32), (0, 0, 0)), ((9, 17, 7), (9 / 16, 17 / 16, 7 / 16), (0, 0, 0)),
         ((24, 8, 25), (0.96, 0.32, 1.0), (0, 0, 0)), ((12, 20, 10), (1, 1, 1), (0, 0, 0)),
         ((10, 14, 12), (1, 1.4, 1.2), (-0.5, 0.25, 1.0)), ((2, 3, 2), (2 / 16, 3 / 16, 2 / 16), (0, 0, 0))]


def particles(n, size, origin, kind, rng):
    size = np.asarray(size)
    h = size / np.asarray(n)
    if kind == "spray":
        pos = rng.uniform(0, 1, (60, 3)) * size
    elif kind == "corners":
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
    pos = np.clip(pos, 0, size) + np.asarray(origin)
    return pos[rng.permutation(len(pos))].astype(np.float32)


def expected(n, size, origin, pos, **kw):
    o = oracle.OracleSim(n, oracle.FLIP, origin=origin, size=size, **kw)
    o.set_particles(pos.astype(np.float64))
    o.stage("sdf")
    return o


@pytest.mark.parametrize("kind", ["block", "spray", "corners", "crowded"])
@pytest.mark.parametrize("n,size,origin", GRIDS)
def test_surface_of_unsorted_particles(n, size, origin, kind):
    pos = particles(n, size, origin, kind, np.random.default_rng(n[0] + len(kind)))
    g = fe.Scene(n, solver=fe.FLIP, size=size, origin=origin, max_cfl=1.0)
    g.set_particles(pos, np.zeros_like(pos))
    o = expected(n, size, origin, pos)
    h = [size[a] / n[a] for a in range(3)]
    mesh = oracle.build_surface(o.sdf(), n, [origin[a] + h[a] / 2.0 for a in range(3)], h)
    for a, b in zip(g.surface(), mesh):
        assert np.array_equal(a, b)
    g.close()


@pytest.mark.parametrize("kind", ["block", "spray", "corners", "crowded"])
@pytest.mark.parametrize("n,size,origin", GRIDS)
def test_viscous_faces_of_sorted_particles(n, size, origin, kind):
    pos = particles(n, size, origin, kind, np.random.default_rng(3 + n[0] + len(kind)))
    g = fe.Scene(n, solver=fe.FLIP, size=size, origin=origin, max_cfl=1.0, viscosity=0.01)
    g.set_particles(pos, np.zeros_like(pos))
    g.run_stages(1 / 240, fe.STAGE_SORT, fe.STAGE_PRE)
    g.run_stages(1 / 240, fe.STAGE_DIFFUSE, fe.STAGE_DIFFUSE)
    o = expected(n, size, origin, pos, viscosity=0.01)
    o.stage("p2g")
    o.stage("diffusion", 1 / 240)
    for a, b in zip(g.diffusion()[1], o.diffusion_markers()):
        assert np.array_equal(a, b)
    g.close()


def test_moved_and_restored_particles():
    """Particles whose cells are not known: the diffusion after a move alone, and the surface after a restore."""
    n, size, origin = GRIDS[0]
    rng = np.random.default_rng(9)
    pos = particles(n, size, origin, "block", rng)
    vel = (rng.standard_normal(pos.shape) * 4).astype(np.float32)
    g = fe.Scene(n, solver=fe.FLIP, size=size, max_cfl=1.0, viscosity=0.01)
    g.set_particles(pos, vel)
    g.step(1 / 240, 1)
    before = g.surface()
    state = g.checkpoint()
    moved = g.particles()[0]
    g.run_stages(1 / 240, fe.STAGE_DIFFUSE, fe.STAGE_DIFFUSE)
    o = expected(n, size, origin, moved, viscosity=0.01)
    o.stage("p2g")
    o.stage("diffusion", 1 / 240)
    for a, b in zip(g.diffusion()[1], o.diffusion_markers()):
        assert np.array_equal(a, b)
    g.step(1 / 240, 2)
    g.restore(state)
    for a, b in zip(g.surface(), before):
        assert np.array_equal(a, b)
    g.close()
