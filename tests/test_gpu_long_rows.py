"""Matrix rows longer than what the solvers hold in shared memory, whose rest is streamed in every
product: dense neighbourhoods (a large radius of 3.1 l0, rows of up to 125 entries) by the one-cluster
solver (72 entries a row at 256 rows a block) and by the resident-matrix solvers with 4, 2 and 1 lanes a
row (96, 48 and 24 entries in FP64, 144, 72 and 36 in FP32), against one launch per kernel.

Every path solves the same system to 1e-12.  The condition numbers of the Jacobi-scaled matrices are
below 2.3 and their diagonals differ by less than a factor of four, so two solutions differ by less
than 2e-12 * 2.3 * 2: 1e-11.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [abi.SOLVER_PLAIN_FP64, abi.SOLVER_MIXED])
@pytest.mark.parametrize("size", [(16, 16, 16), (17, 16, 16), (32, 32, 33), (40, 41, 42)])
def test_rows_past_shared_memory(mps_lib, size, solver):
    from polymps_gb300 import mps
    l0 = 0.01
    fluid = tuple(k * l0 for k in size)
    c = cases.dam3d_polygon(l0=l0, fluid=fluid, tank=(2 * fluid[0] + 0.2, fluid[1], 2 * fluid[2] + 0.2), jitter=0.03)
    c.params.update(reL=3.1)
    with mps.MpsGpu(c, solver=solver, tol=1e-12) as g:
        g.initialize()
        rowptr = g.ppe()[0]
        assert np.diff(rowptr).max() > 100
        out = []
        for mode in (0, 1):
            g.set_ppe_launch(mode)
            g.set(abi.F_PRESSPPE, np.zeros(g.n))
            g.run_op("CALC_PRESS")
            assert g.last_stats().ppeRelResidual <= 1e-12
            out.append(g.get(abi.F_PRESSPPE))
        assert np.any(out[0])
        assert np.linalg.norm(out[1] - out[0]) <= 1e-11 * np.linalg.norm(out[0])
