"""The exchanged words of the reduced solves: a word that never comes ends the solve with an error after a bounded number
of polls, and the words are cleared before their 32-bit tags run over.  The streamed form is reached on a small grid by
refusing the resident form's launch."""
import numpy as np
import pytest

from cms2d_b200 import _lib
from cms2d_b200 import grid as G
from cms2d_b200 import solver as S

pytestmark = pytest.mark.gpu

FORMS = {
    "resident": (dict(precision="fp32_refine", nsolv=3), 0),
    "streamed": (dict(precision="fp32_refine", nsolv=3), 1),
    "bicgstab": (dict(nsolv=3), 0),
    "gmres": (dict(nsolv=4), 0),
}


def _handle(form, g):
    kw, refused = FORMS[form]
    s = S.Solver(g, tol=1e-8, norm=2, **kw)
    _lib.lib().cms_solver_launch_selftest(s._h, refused)
    return s


def _solve(s, system, **kw):
    acoef, ss, sp, phi = [a.copy() for a in system]
    info = s.solve(acoef, ss, sp, np.zeros_like(ss), phi, relax=1.0, nswp=400, **kw)
    return info, phi


@pytest.mark.parametrize("form", list(FORMS))
def test_lost_word_ends_the_solve(form):
    g = G.solver_test_grid(4000)
    system = G.random_system(g, seed=61)
    L = _lib.lib()
    s = _handle(form, g)
    for _ in range(2):  # (a refused launch first gives way to the tiles' form)
        info, ref = _solve(s, system)
        assert info["status"] == _lib.CMS_OK
    assert L.cms_solver_exchange_selftest(s._h, 20000) == _lib.CMS_OK
    info, _ = _solve(s, system, raise_on_error=False)
    assert info["status"] == _lib.CMS_DEVICE_ERROR
    assert "a wait timed out" in L.cms_gpu_last_error().decode()
    # the word restored, the same handle solves as before
    assert L.cms_solver_exchange_selftest(s._h, 0) == _lib.CMS_OK
    info, x = _solve(s, system)
    assert info["status"] == _lib.CMS_OK
    np.testing.assert_array_equal(x, ref)


@pytest.mark.parametrize("form", list(FORMS))
def test_words_are_cleared_before_tags_run_over(form):
    g = G.solver_test_grid(4000)
    system = G.random_system(g, seed=61)
    L = _lib.lib()
    s = _handle(form, g)
    for _ in range(2):
        info, ref = _solve(s, system)
    for room in (5000, 10, 0):  # tags left: one solve's and no second one's, too few, none
        assert L.cms_solver_tag_selftest(s._h, 0xFFFFFFFF - room) == _lib.CMS_OK
        for _ in range(3):
            info, x = _solve(s, system)
            assert info["status"] == _lib.CMS_OK, info
            np.testing.assert_array_equal(x, ref)
    assert L.cms_solver_tag_selftest(s._h, 0) == _lib.CMS_BAD_ARGUMENT
