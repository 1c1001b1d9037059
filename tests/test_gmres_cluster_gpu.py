"""GMRES as one cluster launch against the per-phase kernels: the same bits.

The flow step runs its three systems through it, with fixed caps and loose
tolerances, so an outer iteration that magnifies rounding would show one wrong
bit anywhere in a solve.  Sizes: one partial block, one block, several blocks of the
cluster, rows per thread 1 to 4, matrix and factor in shared memory, matrix
only, neither, two colours and telescoping interfaces; a cycle that ends at its
first or second step (loose tolerances); and a system too large for the
cluster.
"""
import numpy as np
import pytest

from cms2d_b200 import cases
from cms2d_b200.flow import FlowModel

pytestmark = pytest.mark.gpu

CASES = {
    "basin6x5": lambda: cases.tidal_basin(6, 5, seed=3),
    "basin33x31": lambda: cases.tidal_basin(33, 31, seed=3),
    "basin120x100": lambda: cases.tidal_basin(120, 100, seed=4),
    "basin211x177": lambda: cases.tidal_basin(211, 177, seed=5),
    "basin257x255": lambda: cases.tidal_basin(257, 255, seed=6),
    "basin290x270": lambda: cases.tidal_basin(290, 270, seed=7),
    "inlet3k": lambda: cases.tidal_inlet(3_000, seed=1),
    "inlet30k": lambda: cases.tidal_inlet(30_000, seed=2),
    "inlet60k": lambda: cases.tidal_inlet(60_000, seed=3),
}


@pytest.mark.parametrize("kind", list(CASES))
@pytest.mark.parametrize("tol", [1e-3, 0.5, 0.05])
def test_cluster_gmres_bits(kind, tol):
    c = CASES[kind]()
    c.t0 = 0.25 * cases.M2_HOURS * 3600.0
    out = []
    for multi in (True, False):
        m = FlowModel(c, nsolv=4, tol=tol, multi_kernel=multi)
        m.init()
        infos = [m.step() for _ in range(1 if c.grid.ncells > 20_000 else 2)]
        out.append(([m.get(f) for f in ("p", "u", "v")], [(i["niter"], i["krylov_iters"], i["status"]) for i in infos],
                    [s["inner"] for s in m.last_solves()]))
        m.close()
    assert out[0][1:] == out[1][1:]
    for a, b in zip(out[0][0], out[1][0]):
        np.testing.assert_array_equal(a, b)
