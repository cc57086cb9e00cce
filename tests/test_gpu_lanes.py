"""Neighbour sweeps at the edges of their lane split (8, 4 or 1 lanes per particle, by the number
of particles: the lines lie at 12,000 and 40,000), against the FP64 CPU oracle.

The list of the predicted positions is compared bit for bit.  Displacements up to 0.06 spacings
keep the start-of-step skin list (it covers 0.075) while thousands of particles change their
bucket, which are the ones scanned again; 40 spacings make it stale for all of them.  Viscosity
sums of at most 64 terms carry under 100 roundings, so 1e-10 normwise (FP64 tier) and 1e-8
(float-float) hold as for the smaller parity cases.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

from test_gpu_parity import relerr, sync

pytestmark = pytest.mark.gpu

# fluid particles: 36, 11,638 and 12,000, 39,990 and 40,000
SIZES = [(3, 3, 4), (23, 23, 22), (20, 24, 25), (31, 43, 30), (40, 40, 25)]


@pytest.mark.parametrize("kick", [0.06, 40.0])
@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_DF32])
def test_lists_and_viscosity(oracle_mod, mps_lib, size, precision, kick):
    from polymps_gb300 import mps
    l0 = 0.01
    fluid = tuple(k * l0 for k in size)
    c = cases.dam3d_polygon(l0=l0, fluid=fluid, tank=(2 * fluid[0] + 0.2, fluid[1], 2 * fluid[2] + 0.2), jitter=0.03)
    o = oracle_mod.Oracle(c)
    g = mps.MpsGpu(c, precision=precision)
    rng = np.random.default_rng(5)
    o.set(abi.F_VEL, kick * l0 / c.params["timeStep"] * rng.uniform(-0.57, 0.57, (c.n, 3)))
    sync(o, g)
    for ob in (o, g):
        ob.run_op("UPDATE_BUCKETS")
    co, no = o.neighbors()
    cg, ng = g.neighbors()   # built by the scan
    assert np.array_equal(co, cg) and np.array_equal(no, ng)
    for ob in (o, g):
        ob.run_op("VISCOSITY")
    assert relerr(g.get(abi.F_ACC), o.get(abi.F_ACC)) <= (1e-10 if precision == abi.PRECISION_FP64 else 1e-8)
    for ob in (o, g):
        ob.run_op("ADD_GRAVITY")
        ob.run_op("PREDICT")
    o.set(abi.F_POS, g.get(abi.F_POS))   # no field set on the GPU side since the skin list
    co, no = o.neighbors()
    cg, ng = g.neighbors()
    assert np.array_equal(co, cg) and np.array_equal(no, ng)
    g.close()
    o.close()
