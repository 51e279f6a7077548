"""The multigrid levels that one block processes: the limit that a scene reports is the one in effect (the block's shared memory
holds 1612 cells per 256 threads), and the autotuner times no launch choice twice."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

fe = pytest.importorskip("fluide_engine_b200")
from fluide_engine_b200 import autotune  # noqa: E402

DT = 1 / 240


def scene(n):
    size = tuple(k / max(n) for k in n)
    g = fe.Scene(n, solver=fe.FLIP, size=size, max_cfl=1.0, pressure_solver=fe.MGPCG)
    pos, _ = fe.seed_regions([dict(kind=0, lo=(0, 0, 0), hi=(0.4 * size[0], 0.6 * size[1], size[2]))], n, (0, 0, 0), size, 3)
    g.set_particles(pos, np.zeros_like(pos))
    return g


# levels of 32^3: 4096, 512 cells; of 40^3: 8000, 1000, 125; of 20 x 40 x 26: 2600, 350, 60 (10 x 20 x 13, 5 x 10 x 7, 3 x 5 x 4)
@pytest.mark.parametrize("n,threads,cells,effect", [((32, 32, 32), 1024, 4096, 4096), ((32, 32, 32), 512, 4096, 4095),
                                                    ((32, 32, 32), 512, 2048, 2048), ((32, 32, 32), 256, 4096, 4095),
                                                    ((40, 40, 40), 512, 4096, 4096), ((40, 40, 40), 256, 2048, 2048),
                                                    ((20, 40, 26), 512, 4096, 4096), ((20, 40, 26), 256, 4096, 2599),
                                                    ((20, 40, 26), 1024, 2048, 2048)])
def test_reported_limit_is_in_effect(n, threads, cells, effect):
    g = scene(n)
    g.set_tuning(multigrid=1, cg_block_threads=threads, mg_block_level_cells=cells)
    got = g.tuning()
    assert got["mg_block_level_cells"] == effect
    assert all(s["converged"] == 1 for s in g.step(DT, 2))
    g.set_tuning(**got)
    assert g.tuning() == got
    g.set_tuning(cg_block_threads=1024, mg_block_level_cells=cells)
    assert g.tuning()["mg_block_level_cells"] == cells  # a larger block's memory holds them all
    g.close()


@pytest.mark.parametrize("n,candidates", [((32, 32, 32), 3), ((40, 40, 40), 2), ((20, 40, 26), 4)])
def test_no_choice_is_timed_twice(n, candidates):
    g = scene(n)

    def launches(f):
        before = fe.kernel_launch_count()
        f()
        return fe.kernel_launch_count() - before

    per_step = launches(lambda: g.step(DT, 4)) - launches(lambda: g.step(DT, 2))
    tune = lambda k: launches(lambda: autotune.tune(g, DT, substeps=k, save=False, shape_only=True))  # noqa: E731
    assert tune(4) - tune(2) == candidates * per_step
    g.close()
