"""The pressure solvers on either side of the line at which long rows leave the resident matrices (six
million entries streamed a product): just below and above it in the number of rows and in their length,
plain FP64 and mixed, against one launch per kernel.

Every path solves the same system to 1e-12.  The condition numbers of the Jacobi-scaled matrices are
below 2.9 and their diagonals differ by less than a third, so two solutions differ by less than
2e-12 * 2.9 * 1.2: 1e-11.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [abi.SOLVER_PLAIN_FP64, abi.SOLVER_MIXED])
@pytest.mark.parametrize("size,reL", [((47, 47, 48), 2.5), ((48, 48, 49), 2.5), ((39, 39, 40), 3.1), ((42, 42, 41), 3.1)])
def test_solver_beside_the_line(mps_lib, size, reL, solver):
    from polymps_gb300 import mps
    l0 = 0.01
    fluid = tuple(k * l0 for k in size)
    c = cases.dam3d_polygon(l0=l0, fluid=fluid, tank=(2 * fluid[0] + 0.2, fluid[1] + 0.2, 2 * fluid[2] + 0.2), jitter=0.03)
    c.params.update(reL=reL, domainMin=[-0.02] * 3, domainMax=[x + 0.02 for x in c.params["domainMax"]])
    with mps.MpsGpu(c, solver=solver, tol=1e-12) as g:
        g.initialize()
        assert g.n == c.n
        out = []
        for mode in (0, 1):
            g.set_ppe_launch(mode)
            g.set(abi.F_PRESSPPE, np.zeros(c.n))
            g.run_op("CALC_PRESS")
            assert g.last_stats().ppeRelResidual <= 1e-12 and g.last_stats().ppeFallback == 0
            out.append(g.get(abi.F_PRESSPPE))
        assert np.any(out[0])
        assert np.linalg.norm(out[1] - out[0]) <= 1e-11 * np.linalg.norm(out[0])
