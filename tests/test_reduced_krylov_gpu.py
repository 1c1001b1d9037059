"""BiCGStab and GMRES(3) on the rows of groups >= 1 against the per-phase kernels of the same methods.

Both follow the same iterates up to rounding, so the iteration counts agree
and the solutions differ by rounding amplified over the iterations: 1e-11 of
the largest value in FP64 (eps 2e-16 times 5e4), 2e-4 in FP32 (the bound of
the FP32 oracle comparisons; GMRES only, FP32 BiCGStab has its own kernel).  Sizes: a partial slice, one tile and a little
more, one-cell-high grids, islands, telescoping interfaces (rows coupled inside
groups >= 1) on two and three levels, and systems whose vectors and
coefficients fit in shared memory, whose coefficients do not, and whose
vectors do not.
"""
import numpy as np
import pytest

from cms2d_b200 import cases
from cms2d_b200 import grid as G
from cms2d_b200 import solver as S

pytestmark = pytest.mark.gpu


def _islands():
    return G.cartesian_grid(40, 24, 20.0, active=lambda x, y, s: ~(((x > 260) & (x < 300)) | ((y > 200) & (y < 240))))


GRIDS = {
    "3x3": lambda: G.cartesian_grid(3, 3),
    "17x16": lambda: G.cartesian_grid(17, 16),
    "2x300": lambda: G.cartesian_grid(2, 300),
    "40x1": lambda: G.cartesian_grid(40, 1),
    "islands": _islands,
    "tel": lambda: G.solver_test_grid(9000),
    "inlet": lambda: cases.tidal_inlet(12_000).grid,
    "cart600k": lambda: G.cartesian_grid(775, 774),
    "tel1M": lambda: G.solver_test_grid(1_000_000),
    "cart2.2M": lambda: G.cartesian_grid(1483, 1484),
}


@pytest.mark.parametrize("kind", list(GRIDS))
@pytest.mark.parametrize("nsolv, dtype, tol, norm, n", [(3, "float64", 1e-6, 2, 1), (3, "float64", 1e-3, 1, 2),
                                                       (4, "float64", 1e-3, 1, 1), (4, "float64", 1e-6, 1, 2),
                                                       (4, "float32", 1e-3, 1, 2)])
def test_reduced_matches_per_phase_kernels(kind, nsolv, dtype, tol, norm, n):
    g = GRIDS[kind]()
    acoef, ss, sp, phi = G.random_system(g, seed=31, dominance=1.05)
    phi = phi + 0.3 * np.random.default_rng(5).standard_normal(g.ncellsD)  # ghosts included
    acoef, ss, sp, phi = [a.astype(dtype) for a in (acoef, ss, sp, phi)]
    out = []
    for multi in (True, False):
        s = S.Solver(g, tol=tol, norm=norm, nsolv=nsolv, multi_kernel=multi)
        for _ in range(1 if multi else 2):  # the second solve starts from the first one's exchanged words
            a, b, c, p = [x.copy() for x in (acoef, ss, sp, phi)]
            info = s.solve(a, b, c, np.zeros_like(b), p, n=n, nswp=100)
            out.append((info, p))
    (i0, p0), (i1, p1), (i2, p2) = out
    np.testing.assert_array_equal(p1, p2)
    assert (i1["status"], i1["iters"], i1["inner"]) == (i0["status"], i0["iters"], i0["inner"]), (i0, i1)
    assert np.abs(p1 - p0).max() <= (1e-11 if dtype == "float64" else 2e-4) * np.abs(p0).max()
