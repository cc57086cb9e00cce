"""The list sweeps over their options, teacher-forced against the FP64 CPU oracle: radii that
agree and radii that differ (either one the larger), slip and no-slip walls, the gradient types
with and without the correction matrix, and the PND types, at sizes below and above the lines
of the lane split (12,000 and 40,000 particles).

One operator from an identical state, as in the parity tests: sums of at most 128 terms, so
1e-10 normwise in the FP64 tier and 1e-8 in the float-float one.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

from test_gpu_df32 import compare
from test_gpu_parity import step_ops, sync

pytestmark = pytest.mark.gpu

OPTIONS = {
    "radii_equal_grad0": dict(),
    "reL_larger_slip_grad1": dict(reL=2.6, slipCondition=1, gradientType=1),
    "reS_larger_grad2": dict(reS=2.6, gradientType=2),
    "grad3_plain": dict(gradientType=3, gradientCorrection=0),
    "grad3_corrected_mean": dict(gradientType=3, gradientCorrection=1, pndType=1),
    "weight1_grad0": dict(weightType=1, slipCondition=1),
    "wc_diffusive_slip": dict(wc=1, slipCondition=1),
    "wc_diffusive_corrected": dict(wc=1, gradientCorrection=1),
    "wc_shift_velocity": dict(wc=1, shiftingType=1),
}


def _case(opt, size):
    opt = dict(opt)
    l0 = 0.01
    fluid = tuple(k * l0 for k in size)
    c = cases.dam3d_polygon(l0=l0, fluid=fluid, tank=(2 * fluid[0] + 0.2, fluid[1], 2 * fluid[2] + 0.2),
                            jitter=0.03, mode="wc" if opt.pop("wc", 0) else "inc")
    c.params.update(**opt)
    return c


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_DF32])
@pytest.mark.parametrize("size", [(9, 11, 7), (24, 25, 21), (35, 37, 31)])
@pytest.mark.parametrize("name", list(OPTIONS))
def test_sweeps_teacher_forced(oracle_mod, mps_lib, name, size, precision):
    from polymps_gb300 import mps
    c = _case(OPTIONS[name], size)
    o = oracle_mod.Oracle(c)
    o.set_solver(1e-12)
    g = mps.MpsGpu(c, tol=1e-12, precision=precision)
    o.initialize()
    g.initialize()
    rng = np.random.default_rng(3)
    o.set(abi.F_VEL, 0.3 * rng.standard_normal((c.n, 3)))
    o.set_velmax(0.0)   # the GPU has run no corrector yet
    rtol = 1e-10 if precision == abi.PRECISION_FP64 else 1e-8
    sync(o, g)
    for op in step_ops(o.params):
        o.run_op(op)
        g.run_op(op)
        if op == "CALC_PRESS":   # solver paths have their own tests
            sync(o, g)
            continue
        compare(o, g, op, rtol=rtol)
        sync(o, g)
    g.close()
    o.close()
