"""The factor's kernels at the widths and row counts where they can go wrong:
analysis options move the supernode widths over the elimination panels and
the tile edges, and a planted pivot is found wherever it stands in its block.
Backward error 1e-12, the bound of the other solves.  The arithmetic that the
factor's rounding rests on, to the bit."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from temf3dt_b200 import _lib, fetd
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


def test_infinite_diagonal_fixes_its_unknown():
    """An infinite diagonal entry (a Dirichlet condition as a penalty without
    end) gives x = 0 there and the reduced system's solution elsewhere: the
    rows below it are zero (finite / inf), not NaN."""
    m = tiny_synth()
    with _context(m, 96, 2) as g:
        ia, ja, U, A = _matrix(g, 1e-6)
        g.pardiso_alloc(2)
        rng = np.random.default_rng(1)
        fixed = rng.choice(g.n_edges, 7, replace=False)
        va = U.data.copy()
        va[ia[fixed] - 1] = np.inf
        assert g.pardiso_direct_1(1, ia, ja, va) == 0
        free = np.setdiff1d(np.arange(g.n_edges), fixed)
        R = A[free][:, free]
        for cols in (1, 3):
            b = rng.standard_normal((g.n_edges, cols))
            b[free] = R @ b[free]
            x = g.solve(1, b[:, 0] if cols == 1 else b).reshape(g.n_edges, cols)
            assert np.all(x[fixed] == 0.0)
            r = np.linalg.norm(R @ x[free] - b[free], axis=0) / np.linalg.norm(b[free], axis=0)
            assert r.max() <= 1e-12


def _arith(which, n, a, b, out):
    m = tiny_synth()
    with _context(m, 96, 2) as g:
        a, b, out = (np.ascontiguousarray(v, dtype=np.float64) for v in (a, b, out))
        g._ck(_lib.lib().temf_arith_check(g._h, which, n, _lib.dptr(a), _lib.dptr(b), _lib.dptr(out)), "temf_arith_check")
        return out


def test_row_solves_divide_as_the_division_does():
    """Bit for bit, over operands of full mantissas and over those where a
    corrected reciprocal product is hardest: mantissas next to 1 and 2, exact
    quotients, quotients next to a midpoint of two doubles; exponents up to
    the ends of a factor's diagonal and past the range of the corrections;
    zeros of both signs, infinities and NaN."""
    rng = np.random.default_rng(0)
    n = 1 << 19

    def mantissas(k):
        m = 1.0 + rng.random(k)
        e = rng.integers(0, 4, k) * 2.0 ** -52
        return np.where(rng.random(k) < 0.2, np.where(rng.random(k) < 0.5, 1.0 + e, 2.0 - 2.0 ** -52 - e), m)

    a, b = [], []
    for lo, hi in ((-30, 30), (-500, 500)):                   # L_kk = sqrt(d): 2^-537 to 2^512
        den = np.ldexp(mantissas(n), rng.integers(lo, hi, n))
        q = mantissas(n)
        top = np.where(rng.random(n) < 0.4, q * den,          # next to an exact quotient
                       np.where(rng.random(n) < 0.5, q * den + 0.5 * np.spacing(q) * den, mantissas(n) * den))
        a.append(top * np.where(rng.random(n) < 0.5, 1.0, -1.0))
        b.append(den)
    den = np.ldexp(mantissas(n), rng.integers(-537, 512, n))
    a.append(np.ldexp(mantissas(n), rng.integers(-1074, 1023, n)))  # all exponents, denormal to the largest
    b.append(den)
    k = rng.integers(1, 1 << 26, (2, n)).astype(np.float64)   # exact quotients
    a.append(k[0] * k[1])
    b.append(k[1])
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1e308, 1.0])
    a.append(np.repeat(special, 5))
    b.append(np.tile([np.inf, np.nan, 1.0, 2.0 ** 512, 2.0 ** -537], len(special)))
    a, b = np.concatenate(a), np.concatenate(b)
    got = _arith(0, len(a), a, b, np.zeros(len(a)))
    with np.errstate(all="ignore"):
        want = a / b
    same = (got.view(np.uint64) == want.view(np.uint64)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), (a[~same][:4], b[~same][:4], got[~same][:4], want[~same][:4])


def test_dmma_adds_its_products_in_ascending_order():
    """The tiles of the blocks' elimination and of the row solves keep the
    rounding of column-by-column elimination: a DMMA with the target as the
    accumulator is four FMAs, one after the other in ascending k."""
    fma = C.CDLL("libm.so.6").fma
    fma.restype, fma.argtypes = C.c_double, [C.c_double] * 3
    rng = np.random.default_rng(0)
    n = 256
    scale = lambda shape: np.ldexp(rng.standard_normal(shape), rng.integers(-20, 20, shape))
    a, b, c = scale((n, 8, 4)), scale((n, 4, 8)), scale((n, 8, 8))
    got = _arith(1, n, a, b, c.copy()).reshape(n, 8, 8)
    for t in range(n):
        for i in range(8):
            for j in range(8):
                v = c[t, i, j]
                for k in range(4):
                    v = fma(a[t, i, k], b[t, k, j], v)
                assert v == got[t, i, j]


def test_planted_pivot_is_found_at_every_offset_of_a_block():
    """Each of the last 130 columns in elimination order: every position of at
    least one whole 64-column block, in every elimination panel."""
    m = tiny_synth()
    with _context(m, 96, 2) as g:
        ia, ja, U, A = _matrix(g, 1e-6)
        P = A.tocsr()
        P.sort_indices()
        n = g.n_edges
        off = P.indices != np.repeat(np.arange(n), np.diff(P.indptr))
        xadj = np.concatenate([[0], np.cumsum(np.add.reduceat(off, P.indptr[:-1]))]).astype(np.int64)
        adj = P.indices[off].astype(np.int32)
        nod, edg = m.mesh.nod_cor, fetd.mesh_topology(m.mesh.tet_vex)[0]
        mid = np.ascontiguousarray(0.5 * (nod[edg[:, 0] - 1] + nod[edg[:, 1] - 1]))
        perm, st = np.zeros(n, dtype=np.int32), np.zeros(9)
        assert _lib.lib().temf_symbolic_host(n, xadj.ctypes.data_as(C.POINTER(C.c_longlong)), _lib.iptr(adj),
                                             _lib.dptr(mid), _lib.iptr(perm), _lib.dptr(st)) == 0
        assert st[1] == g.stats()["supernodes"]               # the same analysis as the context's
        g.pardiso_alloc(2)
        for col in perm[-130:]:
            va = U.data.copy()
            va[ia[col] - 1] = -10.0 * abs(va[ia[col] - 1])
            assert g.pardiso_direct_1(1, ia, ja, va) == col + 1
