"""The reduced Krylov solves on grids whose first colour has more rows than the later ones together: a block's share of
the group-0 rows then reaches into warps that have no rows of the later groups, and counts in the sums all the same.

Grids with holes (isolated cells and dead ends fall to the first colour), one and several tiles.  After one iteration or
cycle nothing but rounding separates the iterate from the per-phase kernels' (1e-11, as for converged solves), and the
reported ratio in the L2 norm is the true one."""
import numpy as np
import pytest

from cms2d_b200 import grid as G
from cms2d_b200 import solver as S

pytestmark = pytest.mark.gpu


def _holes(nx, ny, share, seed):
    r = np.random.default_rng(seed)
    return G.cartesian_grid(nx, ny, 20.0, active=lambda x, y, s: r.random(np.shape(x)) < share)


GRIDS = {
    "30x20": lambda: _holes(30, 20, 0.45, 1),
    "60x50": lambda: _holes(60, 50, 0.5, 2),
    "200x150": lambda: _holes(200, 150, 0.55, 3),
    "5x1": lambda: G.cartesian_grid(5, 1),
    "77x1": lambda: G.cartesian_grid(77, 1),
}


@pytest.mark.parametrize("kind", list(GRIDS))
@pytest.mark.parametrize("nsolv, norm, nswp", [(3, 2, 1), (3, 1, 1), (3, 2, 4), (4, 2, 1), (4, 2, 3)])
def test_group0_rows_beyond_the_own_rows(kind, nsolv, norm, nswp):
    g = GRIDS[kind]()
    n = g.ncells
    system = G.random_system(g, seed=71)
    out = []
    for multi in (True, False):
        s = S.Solver(g, tol=1e-12, norm=norm, nsolv=nsolv, multi_kernel=multi)
        acoef, ss, sp, phi = [a.copy() for a in system]
        info = s.solve(acoef, ss, sp, np.zeros_like(ss), phi, relax=1.0, nswp=nswp)
        out.append((info, phi[:n]))
    (i0, p0), (i1, p1) = out
    assert (i1["status"], i1["iters"]) == (i0["status"], i0["iters"]), (i0, i1)
    assert np.abs(p1 - p0).max() <= 1e-11 * np.abs(p0).max()
    # (the ratio's own rounding: 1e-11 of the iterate over a residual that has shrunk)
    assert abs(i1["relres"] - i0["relres"]) <= 1e-9 * i0["relres"] + 1e-11, (i0, i1)
