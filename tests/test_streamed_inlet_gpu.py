"""The streamed reduced solve on an inlet whose extended halos are not symmetric (two tiles of the 2.0M-cell inlet
share an edge that only one of them reads): the stopping test's 1e-10 by the FP64 residual, the same bits from a
second solve (which starts from the first one's exchanged words), and the solution of the 1024 x 2 layout.  The
last bound is that of the resident form's tests: residuals of 1e-10 and |A^-1| at most 250, relative to |x|_max."""
import numpy as np
import pytest

from cms2d_b200 import cases
from cms2d_b200 import grid as G
from cms2d_b200 import solver as S

pytestmark = pytest.mark.gpu


def test_streamed_solve_on_one_way_halos():
    g = cases.tidal_inlet(2_000_000).grid
    acoef, ss, sp, phi = G.random_system(g, seed=23)
    out = []
    for lay, calls in ((0, 2), (5, 1)):
        s = S.Solver(g, precision="fp32_refine", tol=1e-10, norm=2, nsolv=3, reduced_layout=lay)
        for _ in range(calls):
            b, p = ss.copy(), phi.copy()
            info = s.solve(acoef, b, sp, np.zeros_like(b), p, relax=1.0, nswp=600)
            assert info["status"] == 0 and info["true_relres"] <= 1e-10, info
            out.append(p[: g.ncells].copy())
        s.close()
    np.testing.assert_array_equal(out[0], out[1])
    assert np.abs(out[0] - out[2]).max() <= 2 * 1e-10 * 250 * np.sqrt(g.ncells) * np.abs(out[2]).max()
