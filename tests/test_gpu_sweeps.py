"""The triangular sweeps at the edges of their layouts: column counts around
the 16-, 32- and 64-column layouts of the block sweeps, supernode widths around
the substitution's panels, and every way the single-column tasks are handed
out (claimed ahead, through the ready queue, by run leaders, subtrees below).
Backward error 1e-12, the bound of the other solves."""
import numpy as np
import pytest

from temf3dt_b200 import fetd
from tests.golden_cases import small_synth, tiny_synth
from tests.test_gpu_factor import _context, _matrix

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(8, 0), (96, 2), (400, 3)])
def factored(request):
    with _context(tiny_synth(), *request.param) as g:
        assert g.factor(1, 2e-6) == 0
        yield g, _matrix(g, 2e-6)[3]


def _worst(A, x, b):
    return float((np.linalg.norm(A @ x - b, axis=0) / np.linalg.norm(b, axis=0)).max())


@pytest.mark.parametrize("cols", [2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 129])
def test_block_sweep_column_counts(factored, cols):
    g, A = factored
    b = A @ np.random.default_rng(cols).standard_normal((g.n_edges, cols))
    assert _worst(A, g.solve(1, b), b) <= 1e-12


@pytest.mark.parametrize("level,split,leaders", [(0, 0, False), (0, 0, True), (0, 4, False), (0, 4, True), (2, 2, False),
                                                 (2, 6, True), (3, 1000, False)])
def test_single_column_plans(factored, level, split, leaders):
    g, A = factored
    levels = int(g.stats()["levels"])
    g.set_solve_plan(min(level, levels - 1), min(split, levels), leaders)
    b = A @ np.random.default_rng(split).standard_normal(g.n_edges)
    for _ in range(2):
        assert _worst(A, g.solve(1, b)[:, None], b[:, None]) <= 1e-12


def test_a_new_analysis_is_untuned():
    """What was tuned on one mesh does not stand for the next one in the same
    context, for one column or for several."""
    with _context(tiny_synth(), 96, 2) as g:
        assert g.factor(1, 2e-6) == 0
        for cols in (1, 5):
            g.tune_solve(1, cols)
            assert g.solve_schedule(cols)[1]
        m = small_synth()
        edg, te, td = fetd.mesh_topology(m.mesh.tet_vex)
        g.set_mesh(m.mesh.nod_cor, m.mesh.tet_vex, edg, te, td)
        g.set_media(*fetd.meshio.media_per_tet(m.mesh.tet_phy, m.ctl))
        g.set_boundary(0)
        g.analyse()
        assert not g.solve_schedule(1)[1] and not g.solve_schedule(5)[1] and not g.solve_plan()["tuned"]
        g.assemble()
        assert g.factor(1, 2e-6) == 0
        A = _matrix(g, 2e-6)[3]
        for cols in (1, 5):
            b = A @ np.random.default_rng(cols).standard_normal((g.n_edges, cols))
            assert _worst(A, g.solve(1, b).reshape(b.shape), b) <= 1e-12
            g.tune_solve(1, cols)
            assert g.solve_schedule(cols)[1]
