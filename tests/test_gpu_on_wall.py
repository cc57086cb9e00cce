"""The wall term of the pressure gradient for a fluid particle that lies exactly on a polygon wall, where
its own image is at distance zero: with gradient type 3 and no particle number density the image's
weight alone multiplies the zero vector, and the weights of types 3 and 4 are finite there.  Against
the FP64 CPU oracle, teacher-forced: 1e-10 normwise in the FP64 tier, 1e-8 in the float-float one.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

from test_gpu_parity import relerr, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_DF32])
@pytest.mark.parametrize("weight", [3, 4])
def test_particle_on_the_wall(oracle_mod, mps_lib, weight, precision):
    from polymps_gb300 import mps
    c = cases.dam3d_polygon(l0=0.01, fluid=(0.12, 0.11, 0.13), tank=(0.4, 0.11, 0.4), jitter=0.03)
    c.params.update(weightType=weight, gradientType=3, gradientCorrection=0)
    o = oracle_mod.Oracle(c)
    g = mps.MpsGpu(c, tol=1e-12, precision=precision)
    o.set_solver(1e-12)
    o.initialize()
    g.initialize()
    o.set_velmax(0.0)   # the GPU has run no corrector yet
    pos = o.get(abi.F_POS)
    i = int(np.argmin(pos[:, 2]))
    pos[i, 2] = 0.0
    o.set(abi.F_POS, pos)
    sync(o, g)
    for op in ("UPDATE_BUCKETS", "WALL_DISTANCE", "WALL_NPCD", "PND_NEIGH_NPCD"):
        o.run_op(op)
        g.run_op(op)
    assert o.get(abi.F_NEARWALL)[i] == 1
    mirror = o.get(abi.F_MIRROR)   # (the closest point may be off by a rounding error)
    mirror[i] = pos[i]
    o.set(abi.F_MIRROR, mirror)
    o.set(abi.F_PNDI, np.zeros(o.n))
    o.set(abi.F_PRESS, np.linspace(0, 1e3, o.n))
    sync(o, g)
    for op in ("PRESS_GRADIENT", "WALL_PRESS_GRADIENT"):
        o.run_op(op)
        g.run_op(op)
        a, b = g.get(abi.F_ACC), o.get(abi.F_ACC)
        assert np.any(b) and np.isfinite(b).all()
        assert relerr(a, b) <= (1e-10 if precision == abi.PRECISION_FP64 else 1e-8)
    g.close()
    o.close()
