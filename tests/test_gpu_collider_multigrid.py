"""Pressure solves with colliders by the multigrid-preconditioned CG: walls inside the domain on even, odd and flat grids
against the plain CG on the same particles (both stop on the same FP64 residual, 1e-9 of the right-hand side, so pressures
agree to that times the system's condition number, below 1e4: 1e-5), and fluid that a collider shuts in, which the plain CG
solves (the same iterations as with the multigrid solver switched off)."""
import numpy as np
import pytest

from meshes import box, icosphere, with_face_normals

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")

BOX = with_face_normals(*box((0.45, -0.1, 0.3), (0.7, 0.35, 0.7)))
BALL = with_face_normals(*icosphere((0.3, 0.25, 0.6), 0.15, 1))
SHEET = with_face_normals(*box((0.28, -0.1, -0.1), (0.34, 0.4, 1.1)))   # about a cell thick, fluid on both sides
LID = with_face_normals(*box((-0.1, 0.25, -0.1), (1.1, 0.4, 1.1)))


def scene(n, meshes, regions, multigrid):
    pos, _ = fe.seed_regions(regions, n, (0, 0, 0), (1, 1, 1), 5)
    for V, _, _ in meshes:  # no particles within the obstacles' bounds: their cells are BOUNDRY
        lo, hi = np.min(V, axis=0), np.max(V, axis=0)
        pos = pos[~np.all((pos > lo) & (pos < hi), axis=1)]
    rng = np.random.default_rng(5)
    g = fe.Scene(n, solver=fe.FLIP, max_cfl=1.0, cg_rel_tol=1e-9)
    for V, T, N in meshes:
        g.add_mesh_collider(V, T, N, n, (0.0, 0.0, 0.0), tuple(1.0 / k for k in n))
    g.set_tuning(multigrid=multigrid)
    g.set_particles(pos, (rng.standard_normal(pos.shape) * 0.4).astype(np.float32))
    return g


@pytest.mark.parametrize("n", [(24, 24, 24), (33, 17, 21), (40, 24, 9), (64, 48, 56)])
@pytest.mark.parametrize("meshes", [[BOX], [BALL], [SHEET], [BOX, BALL]])
def test_pressure_matches_plain_solver(n, meshes):
    out = []
    for multigrid in (0, 1):
        g = scene(n, meshes, [dict(kind=0, lo=(0, 0, 0), hi=(0.8, 0.6, 1.0))], multigrid)
        st = g.step(1 / 240, 1)[0]
        assert st["converged"] == 1 and st["rel_residual"] <= 1e-9
        out.append(g.grid())
        g.close()
    assert np.array_equal(out[0][4], out[1][4])
    if meshes[0] is BOX:  # (the others are thinner than a cell on some of the grids)
        assert (out[0][4] == 2).any()
    for a, b in zip(out[1][:4], out[0][:4]):
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)


def test_shut_in_fluid_is_solved_by_the_plain_solver():
    its = []
    for multigrid in (0, 1):
        g = scene((24, 24, 24), [LID], [dict(kind=0, lo=(0, 0, 0), hi=(1, 0.22, 1)),
                                        dict(kind=0, lo=(0, 0.45, 0), hi=(0.4, 0.8, 1.0))], multigrid)
        st = g.step(1 / 240, 1)[0]
        assert st["converged"] == 1
        its.append(st["cg_iterations"])
        g.close()
    assert abs(its[0] - its[1]) <= 2  # sums in another order
