"""A small radius larger than the large one (reS = 2.6 l0, reL = 2.1 l0): the mirror-side test has to
be made wherever the mirror lies within twice the larger radius of a particle.  Particles in strong
motion, so that some sit between 1.1 times the two radii from the wall with neighbours on the far side
of the mirror's midplane.  Teacher-forced against the FP64 CPU oracle: 1e-10 normwise in the FP64 tier,
1e-8 in the float-float one.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

from test_gpu_df32 import compare
from test_gpu_parity import step_ops, sync

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_DF32])
@pytest.mark.parametrize("opt", [dict(pndType=1), dict(gradientCorrection=1)])
def test_mirror_side_within_the_larger_radius(oracle_mod, mps_lib, opt, precision):
    from polymps_gb300 import mps
    c = cases.dam3d_polygon(l0=0.01, fluid=(0.24, 0.24, 0.24), tank=(0.34, 0.29, 0.34), jitter=0.03)
    c.params.update(reS=2.6, reL=2.1, domainMin=[-0.03] * 3, domainMax=[0.37, 0.32, 0.37], **opt)
    o = oracle_mod.Oracle(c)
    o.set_solver(1e-12)
    g = mps.MpsGpu(c, tol=1e-12, precision=precision)
    o.initialize()
    g.initialize()
    rng = np.random.default_rng(3)
    o.set(abi.F_VEL, 5.0 * rng.standard_normal((c.n, 3)))
    o.set_velmax(0.0)   # the GPU has run no corrector yet
    rtol = 1e-10 if precision == abi.PRECISION_FP64 else 1e-8
    sync(o, g)
    for op in ["UPDATE_BUCKETS", "PREDICT"] + step_ops(o.params):
        o.run_op(op)
        g.run_op(op)
        if op != "CALC_PRESS":   # solver paths have their own tests
            compare(o, g, op, rtol=rtol)
        sync(o, g)
    g.close()
    o.close()
