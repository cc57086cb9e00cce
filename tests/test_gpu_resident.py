"""The resident-matrix pressure solvers at the edges of their row split: the largest systems of
4, 2 and 1 lanes per row on 152 blocks of 768 threads (29,184, 58,368 and 116,736 rows), one
layer more, sizes that leave blocks unevenly filled, and a few rows, against one launch per
kernel.  Every path solves the same system to 1e-12; the matrices' condition numbers after the
Jacobi scaling are below 500, so two solutions differ by less than 1e-9.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu

SIZES = [(4, 3, 3), (7, 5, 11), (48, 38, 16), (49, 38, 16), (48, 38, 32), (47, 39, 33), (48, 38, 64), (49, 38, 64)]


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("solver", [abi.SOLVER_PLAIN_FP64, abi.SOLVER_MIXED])
def test_resident_solvers_agree(mps_lib, size, solver):
    from polymps_gb300 import mps
    l0 = 0.01
    fluid = tuple(k * l0 for k in size)
    c = cases.dam3d_polygon(l0=l0, fluid=fluid, tank=(2 * fluid[0] + 0.2, fluid[1], 2 * fluid[2] + 0.2), jitter=0.03)
    with mps.MpsGpu(c, solver=solver, tol=1e-12) as g:
        g.initialize()
        out = []
        for mode in (0, 1):
            g.set_ppe_launch(mode)
            g.set(abi.F_PRESSPPE, np.zeros(c.n))
            g.run_op("CALC_PRESS")
            assert g.last_stats().ppeRelResidual <= 1e-12
            out.append(g.get(abi.F_PRESSPPE))
        assert np.any(out[0])
        assert np.linalg.norm(out[1] - out[0]) <= 1e-9 * np.linalg.norm(out[0])
