"""The pressure solvers with the right-hand side scaled by 2^30 and 2^-30 (through relaxPND, which
the source is proportional to): by the one-cluster solver, the resident-matrix solvers and the
ones with their vectors in shared memory.  CG is invariant to the scale, and the grid sums hold it
(|r|^2 between 1e-28 and 1e35), so the iteration counts agree to one and the solutions, each of a
system with a condition number below 500 solved to 1e-12, to 1e-9.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("solver", [abi.SOLVER_PLAIN_FP64, abi.SOLVER_MIXED])
@pytest.mark.parametrize("mode", [1, 4])
@pytest.mark.parametrize("size", [(7, 11, 9), (21, 20, 20), (35, 37, 31)])
def test_solution_scales_with_the_source(mps_lib, size, mode, solver):
    from polymps_gb300 import mps
    l0 = 0.01
    fluid = tuple(k * l0 for k in size)
    out, its = [], []
    for scale in (1.0, 2.0 ** 30, 2.0 ** -30):
        c = cases.dam3d_polygon(l0=l0, fluid=fluid, tank=(2 * fluid[0] + 0.2, fluid[1], 2 * fluid[2] + 0.2), jitter=0.03)
        c.params.update(relaxPND=0.01 * scale)
        with mps.MpsGpu(c, solver=solver, tol=1e-12) as g:
            g.set_ppe_launch(mode)
            g.initialize()
            g.set(abi.F_PRESSPPE, np.zeros(c.n))
            g.run_op("CALC_PRESS")
            st = g.last_stats()
            assert st.ppeRelResidual <= 1e-12 and st.ppeFallback == 0
            out.append(g.get(abi.F_PRESSPPE) / scale)
            its.append(st.ppeIterations)
    assert np.any(out[0])
    for k in (1, 2):
        assert abs(its[k] - its[0]) <= 1
        assert np.linalg.norm(out[k] - out[0]) <= 1e-9 * np.linalg.norm(out[0])
