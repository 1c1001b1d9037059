"""The reduced solves (FP64 BiCGStab, GMRES(3), refinement's inner solve) at the ends of their ranges."""
import numpy as np
import pytest

from cms2d_b200 import grid as G
from cms2d_b200 import solver as S
from tests.helpers import interior_matrix

pytestmark = pytest.mark.gpu


def _solve(s, system, scale=1.0, **kw):
    acoef, ss, sp, phi = [a.copy() for a in system]
    ss *= scale
    info = s.solve(acoef, ss, sp, np.zeros_like(ss), phi, relax=1.0, **kw)
    return info, phi


@pytest.mark.parametrize("power", [400, 500, 506])
def test_bicgstab_scales_with_its_right_hand_side(power):
    """The recurrence is homogeneous and its added constants (1e-15) vanish in a right-hand side above 2^300, so scaling
    by a power of two scales every number of the solve exactly: at 2^506 the squared sums are about 2^1022."""
    g = G.cartesian_grid(33, 31)
    system = G.random_system(g, seed=31)
    s = S.Solver(g, tol=1e-8, norm=2, nsolv=3)
    i0, p0 = _solve(s, system, 2.0 ** 300, nswp=300)
    i1, p1 = _solve(s, system, 2.0 ** power, nswp=300)
    assert i0["status"] == 0 and (i1["status"], i1["iters"]) == (0, i0["iters"]), (i0, i1)
    np.testing.assert_array_equal(p1, p0 * 2.0 ** (power - 300))


@pytest.mark.parametrize("layout", [0, 5])
@pytest.mark.parametrize("bad", [1e160, np.inf, np.nan])
def test_refinement_of_a_residual_without_finite_norm_leaves_phi(layout, bad):
    """A residual whose squares overflow, or that is not finite itself, is reported and phi comes back as it went in."""
    g = G.cartesian_grid(33, 31)
    acoef, ss, sp, phi = G.random_system(g, seed=31)
    phi[: g.ncells] = np.random.default_rng(7).standard_normal(g.ncells)
    ss[g.ncells // 2] = bad
    s = S.Solver(g, precision="fp32_refine", tol=1e-8, norm=2, nsolv=3, reduced_layout=layout)
    info, out = _solve(s, (acoef, ss, sp, phi), nswp=300)
    assert info["status"] == 2, info  # CMS_NONFINITE
    np.testing.assert_array_equal(out, phi)


@pytest.mark.parametrize("kind", ["c33", "tel9k"])
@pytest.mark.parametrize("nsolv, nswp", [(3, 1), (3, 2), (3, 7), (4, 1), (4, 2)])
def test_capped_solves_match_per_phase_kernels(kind, nsolv, nswp):
    """The cap ends the solve unconverged on the same iterate: rounding (2e-16) amplified by at most 5e4 over the
    iterations, as for converged solves."""
    g = G.cartesian_grid(33, 31) if kind == "c33" else G.solver_test_grid(9000)
    system = G.random_system(g, seed=33)
    (i0, p0), (i1, p1) = [_solve(S.Solver(g, tol=1e-12, norm=2, nsolv=nsolv, multi_kernel=m), system, nswp=nswp)
                          for m in (True, False)]
    assert i0["status"] == 1  # CMS_NOT_CONVERGED
    assert (i1["status"], i1["iters"], i1["inner"]) == (1, i0["iters"], i0["inner"]) and i1["iters"] == nswp
    assert np.abs(p1 - p0).max() <= 1e-11 * np.abs(p0).max()


@pytest.mark.parametrize("kind", ["c33", "tel9k"])
@pytest.mark.parametrize("tol", [1e-10, 1e-12, 1e-14])
def test_bicgstab_true_residual_at_tight_tolerances(kind, tol):
    """The stopping test is on the recurrence's residual.  An iteration adds at most about 10 u |A||x| of rounding to its
    distance from b - A x (u = 2^-53; a row has at most 7 entries and the update of x two more roundings).  Whether the
    tolerance is met is the method's own matter (its added constants of 1e-15 stop it near 1e-10 here): as the per-phase
    kernels."""
    g = G.cartesian_grid(33, 31) if kind == "c33" else G.solver_test_grid(9000)
    system = G.random_system(g, seed=33)
    (i0, _), (info, phi) = [_solve(S.Solver(g, tol=tol, norm=2, nsolv=3, multi_kernel=m), system, nswp=300)
                            for m in (True, False)]
    assert (info["status"], info["iters"]) == (i0["status"], i0["iters"])
    n = g.ncells
    A = interior_matrix(g, system[0], system[2])
    b, x = system[1][:n], phi[:n]
    size = np.linalg.norm(abs(A) @ np.abs(x)) / np.linalg.norm(b)
    true = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
    assert abs(true - info["relres"]) <= 10 * 2.0 ** -53 * info["iters"] * size, (true, info)
