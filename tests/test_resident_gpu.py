"""The resident form of the reduced inner solve (reduced_layout 0) at the edges of its tiles.

Sizes: a single partial slice of 32 rows, one tile, tiles cut just below and
above a multiple of the rows per tile, a strip narrower than a tile, islands
(a grid in several pieces), telescoping interfaces, two and four rows per
thread, and systems too large for the SMs (the streamed form, with all, some and none
of its vectors in shared memory).  Each
solution is compared with a direct FP64 solve; the stopping test asks for a
1e-10 residual, |A^-1| is at most 1 / (0.02 * 0.2) = 250 (diagonal 1.02 times
a row sum of at least two coefficients of 0.1) and |b| / |x|_max at most
sqrt(n) here, so 1e-10 * 250 * sqrt(n) bounds the error relative to |x|_max
(right-hand side and solution of order one).
"""
import numpy as np
import pytest

from cms2d_b200 import grid as G
from cms2d_b200 import solver as S
from tests.helpers import interior_matrix

pytestmark = pytest.mark.gpu


def _islands():
    return G.cartesian_grid(40, 24, 20.0, active=lambda x, y, s: ~(((x > 260) & (x < 300)) | ((y > 200) & (y < 240))))


GRIDS = {
    "5x5": lambda: G.cartesian_grid(5, 5),
    "8x8": lambda: G.cartesian_grid(8, 8),
    "16x15": lambda: G.cartesian_grid(16, 15),
    "17x16": lambda: G.cartesian_grid(17, 16),
    "2x300": lambda: G.cartesian_grid(2, 300),
    "300x2": lambda: G.cartesian_grid(300, 2),
    "islands": _islands,
    "tel": lambda: G.solver_test_grid(9000),
}


def _solve(g, seed, **kw):
    acoef, ss, sp, phi = G.random_system(g, seed=seed)
    phi = phi.copy()
    phi[g.ncells:] = np.random.default_rng(seed).standard_normal(g.ncellsD - g.ncells)  # ghost values enter the rhs
    s = S.Solver(g, precision="fp32_refine", tol=1e-10, norm=2, nsolv=3, **kw)
    out = []
    for _ in range(2):  # the second call starts from the first one's exchanged words
        a, b, c, p = [x.copy() for x in (acoef, ss, sp, phi)]
        info = s.solve(a, b, c, np.zeros_like(b), p, relax=1.0, nswp=600)
        assert info["status"] == 0, info
        out.append((info, p[: g.ncells].copy()))
    np.testing.assert_array_equal(out[0][1], out[1][1])
    return acoef, ss, sp, phi, out[0]


@pytest.mark.parametrize("kind", list(GRIDS))
def test_resident_matches_direct_solve(kind):
    import scipy.sparse.linalg as spla
    g = GRIDS[kind]()
    n = g.ncells
    acoef, ss, sp, phi, (info, x) = _solve(g, 21)
    A = interior_matrix(g, acoef, sp)
    rhs = ss[:n].copy()
    for k in range(g.nmaxfaces):
        c = g.cell2cell[:n, k]
        m = (k < g.ncface[:n]) & (c > n)
        rhs[m] += acoef[:n, k][m] * phi[c[m] - 1]
    ref = spla.spsolve(A.tocsc(), rhs)
    assert np.abs(x - ref).max() <= 1e-10 * 250 * np.sqrt(n) * np.abs(ref).max(), info


@pytest.mark.parametrize("kind, cells", [("cart", 330_000), ("tel", 500_000), ("cart", 1_160_000), ("cart", 1_300_000),
                                         ("tel", 2_000_000), ("cart", 5_600_000)])
def test_resident_rows_per_thread(kind, cells):
    """Two, four and eight rows per thread, and the streamed form beyond: the
    FP64 residual of the result, and the solution of the 1024 x 2 layout."""
    side = int(round(cells ** 0.5))
    g = G.cartesian_grid(side, side) if kind == "cart" else G.solver_test_grid(cells)
    *_, (info, x) = _solve(g, 22)
    *_, (_, y) = _solve(g, 22, reduced_layout=5)
    assert info["true_relres"] <= 1e-10
    assert np.abs(x - y).max() <= 2 * 1e-10 * 250 * np.sqrt(g.ncells) * np.abs(y).max()
