"""Connectivities with one-way couplings (a cell lists a neighbour that does not list it): the multicolour groups are then
not independent, so the forms that take group 0 as independent stay out: GMRES runs its per-phase kernels, some 25
launches per cycle, and builds no tables."""
import numpy as np
import pytest

from cms2d_b200 import grid as G
from cms2d_b200 import solver as S

pytestmark = pytest.mark.gpu


def _grid(seed):
    """A Cartesian grid of which every tenth cell has lost its last two faces, those to earlier cells, so that half of
    these cells get the colour of cells that list them."""
    g = G.cartesian_grid(40, 30)
    c2c, nf = g.cell2cell.copy(), g.ncface.copy()
    for i in np.random.default_rng(seed).choice(g.ncells, g.ncells // 10, replace=False):
        nf[i] -= min(2, nf[i])
        c2c[i, nf[i]:] = 0
    return G.Grid(ncells=g.ncells, ncellsD=g.ncellsD, nmaxfaces=g.nmaxfaces, cell2cell=c2c, ncface=nf,
                  idirface=g.idirface, x=g.x, y=g.y, dx=g.dx, dy=g.dy, level=g.level, telescoping=g.telescoping)


@pytest.mark.parametrize("one_way", [True, False])
@pytest.mark.parametrize("precision, dtype", [("fp64", "float64"), ("fp64", "float32"), ("fp32_refine", "float64")])
def test_forms_for_independent_groups_stay_out(one_way, precision, dtype):
    import torch
    g = _grid(1) if one_way else G.cartesian_grid(40, 30)
    acoef, ss, sp, phi = [torch.from_numpy(a.astype(dtype)).cuda() for a in G.random_system(g, seed=1, dominance=1.05)]
    s = S.Solver(g, precision=precision, tol=1e-12, nsolv=4)
    held, launched = s.device_bytes, s.launches
    info = s.solve(acoef, ss, sp, torch.zeros_like(ss), phi, relax=1.0, nswp=4)
    assert (s.launches - launched > 20 * info["inner"] / 3) == one_way, info  # three Arnoldi steps per cycle
    assert (s.device_bytes == held) == (one_way or precision == "fp32_refine")
