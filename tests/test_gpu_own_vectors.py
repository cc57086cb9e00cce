"""The mixed pressure solver with four, three or two of its inner vectors in shared memory (by the
rows of a block; MPSGPU_OWN_VECTORS, read when a handle is created, sets the number), at the
first size above the resident-matrix solvers and one that leaves a remainder round, against one
launch per kernel.  All solve the same system to 1e-12; the matrices' condition numbers after
the Jacobi scaling are below 500, so two solutions differ by less than 1e-9.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(49, 48, 50), (61, 59, 53)])
@pytest.mark.parametrize("vectors", ["4", "3", "2"])
def test_vectors_in_shared_memory(mps_lib, size, vectors, monkeypatch):
    from polymps_gb300 import mps
    monkeypatch.setenv("MPSGPU_OWN_VECTORS", vectors)
    l0 = 0.01
    fluid = tuple(k * l0 for k in size)
    c = cases.dam3d_polygon(l0=l0, fluid=fluid, tank=(2 * fluid[0] + 0.2, fluid[1], 2 * fluid[2] + 0.2), jitter=0.03)
    with mps.MpsGpu(c, solver=abi.SOLVER_MIXED, tol=1e-12) as g:
        g.initialize()
        out = []
        for mode in (0, 1):
            g.set_ppe_launch(mode)
            g.set(abi.F_PRESSPPE, np.zeros(c.n))
            g.run_op("CALC_PRESS")
            assert g.last_stats().ppeRelResidual <= 1e-12 and g.last_stats().ppeFallback == 0
            out.append(g.get(abi.F_PRESSPPE))
        assert np.linalg.norm(out[1] - out[0]) <= 1e-9 * np.linalg.norm(out[0])
