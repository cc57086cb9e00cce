"""The one-cluster pressure solver (plain FP64, up to 4,096 rows) at the edges of its shape: a few
rows on one of its blocks, whole warps, rows that do not fill the last block, the last row count
it takes and the next above it, against one launch per kernel.  Both solve the same system to 1e-12; the matrices' condition numbers after
the Jacobi scaling are below 500, so two solutions differ by less than 1e-9.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (4, 4, 32), (7, 11, 9), (13, 17, 17), (16, 16, 16), (17, 13, 19)]


@pytest.mark.parametrize("size", SIZES)
def test_cluster_solver(mps_lib, size):
    from polymps_gb300 import mps
    l0 = 0.01
    fluid = tuple(k * l0 for k in size)
    c = cases.dam3d_polygon(l0=l0, fluid=fluid, tank=(2 * fluid[0] + 0.2, fluid[1], 2 * fluid[2] + 0.2), jitter=0.03)
    with mps.MpsGpu(c, tol=1e-12) as g:
        g.initialize()
        out, its = [], []
        for mode in (0, 1):
            g.set_ppe_launch(mode)
            g.set(abi.F_PRESSPPE, np.zeros(c.n))
            g.run_op("CALC_PRESS")
            st = g.last_stats()
            assert st.ppeRelResidual <= 1e-12
            out.append(g.get(abi.F_PRESSPPE))
            its.append(st.ppeIterations)
        assert abs(its[0] - its[1]) <= 1
        assert np.linalg.norm(out[1] - out[0]) <= 1e-9 * np.linalg.norm(out[0])
        # from the solution: nothing left to do, the result stands
        g.run_op("CALC_PRESS")
        assert g.last_stats().ppeRelResidual <= 1e-12


def test_iteration_cap_is_reported(mps_lib):
    from polymps_gb300 import mps
    c = cases.dam3d_polygon(l0=0.01, fluid=(0.1, 0.1, 0.1), tank=(0.4, 0.1, 0.4), jitter=0.03)
    with mps.MpsGpu(c) as g:
        g.initialize()
        g.set(abi.F_PRESSPPE, np.zeros(c.n))
        g.set_solver(tol=1e-12, max_iter=3)
        with pytest.raises(mps.MpsError):
            g.run_op("CALC_PRESS")
        assert g.last_stats().ppeIterations == 3
