"""Signs of a closed mesh whose surface runs through many of the grid's nodes, which sum the winding terms of all triangles
themselves: against the oracle at counts where that sum takes from one to 32 lanes a node, and not slower than the same mesh
with a triangle missing, of which every node sums."""
import time

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")

ZERO = (0.0, 0.0, 0.0)


def box(n, h, cells):
    """The grid's own box, `cells` squares along each edge, outward triangles (V, T)."""
    hi = (np.asarray(n) - 1) * h
    V, T = [], []
    for a in range(3):
        u, v = (a + 1) % 3, (a + 2) % 3
        for side in (0, 1):
            base = len(V)
            for i in range(cells + 1):
                for j in range(cells + 1):
                    p = np.zeros(3)
                    p[a], p[u], p[v] = side * hi[a], hi[u] * (i / cells), hi[v] * (j / cells)
                    V.append(p)
            for i in range(cells):
                for j in range(cells):
                    q = [base + i * (cells + 1) + j, base + (i + 1) * (cells + 1) + j, base + (i + 1) * (cells + 1) + j + 1,
                         base + i * (cells + 1) + j + 1]
                    q = q if side else q[::-1]
                    T += [(q[0], q[1], q[2], 0), (q[0], q[2], q[3], 0)]
    return np.array(V), np.array(T, dtype=np.int64)


# all or most nodes on the surface: 160 to 320,000 of them
@pytest.mark.parametrize("n,cells", [((40, 2, 2), 4), ((17, 9, 2), 3), ((100, 60, 2), 2), ((33, 33, 33), 2), ((2, 200, 200), 1),
                                     ((400, 400, 2), 1), ((48, 3, 50), 5)])
def test_signs_match_oracle(n, cells):
    h = 1.0 / 32
    V, T = box(n, h, cells)
    assert np.array_equal(fe.mesh_to_sdf(V, T, n, ZERO, (h,) * 3), oracle.mesh_to_sdf(V, T, n, ZERO, (h,) * 3))


@pytest.mark.parametrize("n,cells", [((1024, 2, 2), 32), ((256, 4, 4), 16)])
def test_not_slower_than_an_open_mesh(n, cells):
    h = 1.0 / 64
    V, T = box(n, h, cells)

    def best(T):
        times = []
        for _ in range(4):
            t = time.perf_counter()
            fe.mesh_to_sdf(V, T, n, ZERO, (h,) * 3)
            times.append(time.perf_counter() - t)
        return min(times)

    assert best(T) <= 2.0 * best(T[:-1])


@pytest.mark.parametrize("n", [(16, 16, 16), (65, 64, 64), (7, 90, 4)])
@pytest.mark.parametrize("cells", [1, 2, 3])
def test_few_triangles(n, cells):
    """12, 48 and 108 triangles: either side of the counts from which crossings are recorded; closed and open."""
    h = 1.0 / 32
    V, T = box(n, h, cells)
    V = V * 0.77 + 0.01  # off the nodes
    for triangles in (T, T[:-1]):
        assert np.array_equal(fe.mesh_to_sdf(V, triangles, n, ZERO, (h,) * 3), oracle.mesh_to_sdf(V, triangles, n, ZERO, (h,) * 3))
