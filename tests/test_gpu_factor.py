"""The factor's kernels at the widths and row counts where they can go wrong:
analysis options move the supernode widths over the elimination panels and
the tile edges, and a planted pivot is found wherever it stands in its block.
Backward error 1e-12, the bound of the other solves."""
import numpy as np
import pytest
import scipy.sparse as sp

from temf3dt_b200 import fetd
from tests.golden_cases import tiny_synth

pytestmark = pytest.mark.gpu


def _context(m, leaf, level):
    g = fetd.FetdGPU(0)
    edg, te, td = fetd.mesh_topology(m.mesh.tet_vex)
    g.set_analysis_options(leaf, level)
    g.set_mesh(m.mesh.nod_cor, m.mesh.tet_vex, edg, te, td)
    g.set_media(*fetd.meshio.media_per_tet(m.mesh.tet_phy, m.ctl))
    g.set_boundary(0)
    g.analyse()
    g.assemble()
    return g


def _matrix(g, dt):
    ia, ja, m = g.get_matrix(0)
    _, _, k = g.get_matrix(1)
    U = sp.csr_matrix((3.0 * m + 2.0 * dt * k, ja - 1, ia - 1), shape=(g.n_edges, g.n_edges))
    return ia, ja, U, U + sp.triu(U, 1).T


@pytest.mark.parametrize("leaf,level", [(8, 0), (9, 2), (17, 0), (40, 1), (96, 2), (150, 3), (400, 3)])
def test_factor_at_supernode_widths(leaf, level):
    m = tiny_synth()
    with _context(m, leaf, level) as g:
        rng = np.random.default_rng(leaf)
        for dt in (1e-7, 1e-4):
            assert g.factor(1, dt) == 0
            _, _, _, A = _matrix(g, dt)
            for cols in (1, 3):
                b = A @ rng.standard_normal((g.n_edges, cols))
                x = g.solve(1, b[:, 0] if cols == 1 else b).reshape(g.n_edges, cols)
                r = np.linalg.norm(A @ x - b, axis=0) / np.linalg.norm(b, axis=0)
                assert r.max() <= 1e-12


def test_planted_pivot_is_found_in_every_position():
    m = tiny_synth()
    with _context(m, 96, 2) as g:
        ia, ja, U, A = _matrix(g, 1e-6)
        g.pardiso_alloc(2)
        rng = np.random.default_rng(0)
        for col in rng.choice(g.n_edges, 24, replace=False):
            va = U.data.copy()
            va[ia[col] - 1] = -10.0 * abs(va[ia[col] - 1])    # the diagonal is a row's first entry
            assert g.pardiso_direct_1(1, ia, ja, va) == col + 1
