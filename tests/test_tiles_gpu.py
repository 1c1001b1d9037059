"""The tiles of a handle's FP64 persistent solves do not depend on what the handle has solved in FP32.

Above 151,552 cells FP32 BiCGStab runs as one block per SM, FP64 as four; the sums are added by tiles, so a solve on
other tiles has other bits.  The reduced form that FP64 takes by itself is refused its tables here."""
import numpy as np
import pytest

from cms2d_b200 import _lib
from cms2d_b200 import grid as G
from cms2d_b200 import solver as S

pytestmark = pytest.mark.gpu


def test_fp64_tiles_after_an_fp32_solve():
    import torch
    g = G.cartesian_grid(420, 410)
    system = G.random_system(g, seed=51)
    L = _lib.lib()

    def solve(s, dtype):
        acoef, ss, sp, phi = [torch.from_numpy(a.astype(dtype)).cuda() for a in system]
        info = s.solve(acoef, ss, sp, torch.zeros_like(ss), phi, relax=1.0, nswp=300)
        assert info["status"] == 0, info
        return phi.cpu().numpy()

    out = []
    for fp32_first in (False, True):
        s = S.Solver(g, tol=1e-5, norm=2, nsolv=3)
        if fp32_first:
            single = solve(s, "float32")
        L.cms_solver_alloc_selftest(s._h, 0, 1)
        out.append(solve(s, "float64"))
        if fp32_first:
            np.testing.assert_array_equal(solve(s, "float32"), single)
        s.close()
    np.testing.assert_array_equal(out[0], out[1])
