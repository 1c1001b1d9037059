"""GMRES(3) on the rows of groups >= 1 stops on the residual b - A x, as the per-phase kernels do, also where rounding
separates that from the residual of the recurrence: FP32 at tolerances near its rounding, FP64 at the attainable accuracy.

The true residual, formed here in FP64 from the call's arrays, is compared with the per-phase kernels'.  At a met
tolerance it is made of what the stopping test saw (at most tol) and of the rounding e of the last cycle (its residual's
sums and the update of x), at right angles but for chance; both forms round the same expressions, so e is taken from the
per-phase solve: true <= 1.1 sqrt(tol^2 + e^2).  The norm of independent roundings over n rows spreads by 1/sqrt(n), 3 %
for the smallest grid.  At the attainable accuracy the residual is e alone, of a last cycle that chance picks: 1.5 times
the per-phase one."""
import numpy as np
import pytest

from cms2d_b200 import grid as G
from cms2d_b200 import solver as S
from tests.helpers import interior_matrix

pytestmark = pytest.mark.gpu

GRIDS = {
    "c33": lambda: G.cartesian_grid(33, 31),
    "c200": lambda: G.cartesian_grid(200, 200),
    "tel9k": lambda: G.solver_test_grid(9000),
}


def _solve(g, dominance, dtype, tol, multi):
    system = [a.astype(dtype) for a in G.random_system(g, seed=31, dominance=dominance)]
    acoef, ss, sp, phi = [a.copy() for a in system]
    s = S.Solver(g, tol=tol, nsolv=4, multi_kernel=multi)
    info = s.solve(acoef, ss, sp, np.zeros_like(ss), phi, relax=1.0, nswp=400)
    acoef, ss, sp, _ = [a.astype(np.float64) for a in system]
    n = g.ncells
    A = interior_matrix(g, acoef, sp)
    b = ss[:n]  # (ghost values are 0)
    return info, float(np.linalg.norm(b - A @ phi[:n].astype(np.float64)) / np.linalg.norm(b))


@pytest.mark.parametrize("kind", list(GRIDS))
@pytest.mark.parametrize("dominance", [1.02, 1.002])
@pytest.mark.parametrize("dtype, tol", [("float32", 1e-5), ("float32", 1e-6), ("float64", 1e-6), ("float64", 1e-14)])
def test_true_residual_as_per_phase_kernels(kind, dominance, dtype, tol):
    g = GRIDS[kind]()
    i0, t0 = _solve(g, dominance, dtype, tol, True)
    i1, t1 = _solve(g, dominance, dtype, tol, False)
    assert i1["status"] == i0["status"], (i0, i1)
    if i0["status"] == 0:
        assert t1 <= 1.1 * np.sqrt(tol ** 2 + max(t0 ** 2 - i0["relres"] ** 2, 0.0)), (t0, t1, i0, i1)
    else:
        assert t1 <= 1.5 * t0, (t0, t1, i0, i1)
