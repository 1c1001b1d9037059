"""The ensemble's solves on tiles of 256 threads: more blocks asked for than the device has SMs, or members too large
for the resident form.  Each member's fields follow its own steps, whose solves run in another form, to the solves'
tolerance (1e-7 m and 1e-6 of the largest speed at 1e-8, as for other splits of the batched launch); and a member that
steps on its own between two steps of the ensemble leaves the ensemble's tables usable."""
import numpy as np
import pytest

from cms2d_b200 import cases
from cms2d_b200.ensemble import EnsembleModel
from cms2d_b200.flow import FlowModel

pytestmark = pytest.mark.gpu

SET = dict(precision="fp32_refine", nsolv=3, tol=1e-8, norm=2, nswp_pp=400, nswp_uv=400)


def _one_dt(cs):
    for c in cs:
        c.dt = 300.0  # (an ensemble steps with one)
    return cs


def _fields(m, n):
    return {k: m.get(k)[:n].copy() for k in ("eta", "u", "v")}


def _solo(c, steps):
    m = FlowModel(c, **SET)
    m.init()
    for _ in range(steps):
        assert m.step()["status"] == 0
    out = _fields(m, c.grid.ncells)
    m.close()
    return out


def _compare(m, ref, c):
    got = _fields(m, c.grid.ncells)
    assert np.abs(got["eta"] - ref["eta"]).max() <= 1e-7
    vmax = np.hypot(ref["u"], ref["v"]).max()
    for k in ("u", "v"):
        assert np.abs(got[k] - ref[k]).max() <= 1e-6 * vmax, k


@pytest.mark.parametrize("blocks", [300, 592])
def test_tile_form_matches_member_steps(blocks):
    cs = _one_dt([cases.tidal_basin(220, 120, seed=4, amp=0.6), cases.tidal_inlet(12_000, seed=5),
                  cases.tidal_basin(40, 30, seed=1, amp=0.5)])
    solo = [_solo(c, 2) for c in cs]
    e = EnsembleModel(cs, **SET)
    e.set_tiles(blocks)
    tot, per = e.tiles()
    assert 148 < tot <= blocks and per.min() >= 1
    e.init()
    for _ in range(2):
        infos = e.step()
        assert all(i["status"] == 0 for i in infos), infos
    for m, ref, c in zip(e.members, solo, cs):
        _compare(m, ref, c)
    e.close()


@pytest.mark.parametrize("blocks", [0, 300])
def test_member_steps_on_its_own_in_between(blocks):
    cs = _one_dt([cases.tidal_basin(120, 90, seed=4, amp=0.6), cases.tidal_inlet(9_000, seed=5)])
    ref = []
    for c, own in zip(cs, (True, False)):  # the same water levels on each one's own
        m = FlowModel(c, **SET)
        m.init()
        m.step()
        if own:
            m.step()
            m.t -= c.dt
        m.step()
        ref.append(_fields(m, c.grid.ncells))
        m.close()
    e = EnsembleModel(cs, **SET)
    if blocks:
        e.set_tiles(blocks)
    e.init()
    e.step()
    assert e.members[0].step()["status"] == 0  # its solves build tables for tiles of their own
    infos = e.step()  # (its levels are those of the ensemble's time)
    assert all(i["status"] == 0 for i in infos), infos
    for m, r, c in zip(e.members, ref, cs):
        _compare(m, r, c)
    e.close()
