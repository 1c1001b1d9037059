"""A device allocation or a launch that is refused inside a solve: the solve goes on in the form that does without it, and later
solves of the handle are right too.  The refusal is a request larger than the device, made at every allocation of a
first solve in turn (one refused, and that one and all that follow).

Each solution is compared with the one of a handle that is refused nothing.  Both meet 1e-9 of the first residual,
|A^-1| is at most 250 (diagonal 1.02 times a row sum of at least 0.2) and |b| / |x|_max at most sqrt(n), so they differ
by at most 2 * 1e-9 * 250 * sqrt(n) of the largest value."""
import numpy as np
import pytest

from cms2d_b200 import _lib
from cms2d_b200 import grid as G
from cms2d_b200 import solver as S

pytestmark = pytest.mark.gpu

FORMS = {
    "bicgstab": dict(nsolv=3),
    "gmres": dict(nsolv=4),
    "refinement": dict(nsolv=3, precision="fp32_refine"),  # resident, then streamed, then the tiles' form
}


def _solve(s, g, system, nswp=400):
    import torch
    acoef, ss, sp, phi = [torch.from_numpy(a.copy()).cuda() for a in system]  # (no staging buffers)
    info = s.solve(acoef, ss, sp, torch.zeros_like(ss), phi, relax=1.0, nswp=nswp)
    return info, phi.cpu().numpy()[: g.ncells]


@pytest.mark.parametrize("form", list(FORMS))
def test_refused_allocations(form):
    g = G.solver_test_grid(4000)
    system = G.random_system(g, seed=41)
    kw = dict(tol=1e-9, norm=2, **FORMS[form])
    s = S.Solver(g, **kw)
    info, ref = _solve(s, g, system)
    assert info["status"] == 0
    full = s.device_bytes
    bound = 2 * 1e-9 * 250 * np.sqrt(g.ncells) * np.abs(ref).max()
    s.close()
    L = _lib.lib()
    for count in (1, 1000):
        refused = []
        for first in range(60):
            s = S.Solver(g, **kw)
            L.cms_solver_alloc_selftest(s._h, first, count)
            held = []
            for _ in range(2):  # with the refusal, and without
                info, x = _solve(s, g, system)
                assert info["status"] == 0 and np.abs(x - ref).max() <= bound, (first, count, info)
                held.append(s.device_bytes)
                L.cms_solver_alloc_selftest(s._h, 0, 0)
            refused.append(held[0] != full)
            s.close()
        assert refused[0] and not refused[-1]  # every allocation of the solve had its turn


@pytest.mark.parametrize("count", [1, 2])
def test_refused_launch_of_the_resident_form(count):
    """The refinement finishes in the tiles' form, and later solves of the handle keep to the forms that fit."""
    g = G.solver_test_grid(4000)
    system = G.random_system(g, seed=41)
    kw = dict(tol=1e-9, norm=2, nsolv=3, precision="fp32_refine")
    s = S.Solver(g, **kw)
    _, ref = _solve(s, g, system)
    s.close()
    s = S.Solver(g, **kw)
    _lib.lib().cms_solver_launch_selftest(s._h, count)  # 2: the streamed form's too
    for _ in range(3):
        info, x = _solve(s, g, system)
        assert info["status"] == 0 and info["true_relres"] <= 1e-9, info
        assert np.abs(x - ref).max() <= 2 * 1e-9 * 250 * np.sqrt(g.ncells) * np.abs(ref).max()


@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_no_tables_for_tiles_that_cannot_fit(dtype):
    """Beyond about 8M cells a tile's gathered vector alone exceeds an SM's shared memory: nothing of the reduced forms is
    built or allocated on the way to the form that runs."""
    import torch
    g = G.cartesian_grid(3000, 3001)
    acoef, ss, sp, phi = [torch.from_numpy(a.astype(dtype)).cuda() for a in G.random_system(g, seed=5)]
    s = S.Solver(g, nsolv=4)
    before = s.device_bytes
    info = s.solve(acoef, ss, sp, torch.zeros_like(ss), phi, relax=1.0, nswp=2)
    assert info["iters"] == 2 and s.device_bytes == before
