"""A large radius of 3.1 l0, whose neighbourhoods do not fit the start-of-step list's rows: above the
line of the lane split (40,000 particles) every sweep scans the buckets, below it the overflowing rows
do; and 2.9 l0, whose rows just fit.  Teacher-forced against the FP64 CPU oracle: sums of at
most 128 terms, so 1e-10 normwise in the FP64 tier and 1e-8 in the float-float one.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

from test_gpu_df32 import compare
from test_gpu_parity import step_ops, sync

pytestmark = pytest.mark.gpu

OPTIONS = {
    "inc": dict(),
    "inc_relax": dict(relaxPress=0.5),
    "wc_shift_velocity": dict(wc=1, shiftingType=1),
    "wc_shift_gradient": dict(wc=1, shiftingType=2),
}


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_DF32])
@pytest.mark.parametrize("size,reL", [((36, 37, 35), 3.1), ((36, 37, 35), 2.9), ((12, 13, 11), 3.1)])
@pytest.mark.parametrize("name", list(OPTIONS))
def test_sweeps_with_a_long_radius(oracle_mod, mps_lib, name, size, reL, precision):
    from polymps_gb300 import mps
    opt = dict(OPTIONS[name])
    l0 = 0.01
    fluid = tuple(k * l0 for k in size)
    c = cases.dam3d_polygon(l0=l0, fluid=fluid, tank=(2 * fluid[0] + 0.2, fluid[1] + 0.2, 2 * fluid[2] + 0.2),
                            jitter=0.03, mode="wc" if opt.pop("wc", 0) else "inc")
    # (the reference removes what lies within a bucket of the domain's edge)
    c.params.update(reL=reL, domainMin=[-0.02] * 3, domainMax=[x + 0.02 for x in c.params["domainMax"]], **opt)
    o = oracle_mod.Oracle(c)
    o.set_solver(1e-12)
    g = mps.MpsGpu(c, tol=1e-12, precision=precision)
    o.initialize()
    g.initialize()
    assert o.n == g.n == c.n
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


@pytest.mark.parametrize("reL,launches", [(2.9, 2), (3.1, 1)])
def test_list_only_where_its_rows_hold_the_neighbours(mps_lib, reL, launches):
    """The viscosity is the list's build and a sweep over it, or one scan of the buckets."""
    import ctypes as C
    from polymps_gb300 import mps
    l0 = 0.01
    c = cases.dam3d_polygon(l0=l0, fluid=(0.36, 0.37, 0.35), tank=(0.92, 0.57, 0.9), jitter=0.03)
    c.params.update(reL=reL, domainMin=[-0.02] * 3, domainMax=[0.94, 0.59, 0.92])
    with mps.MpsGpu(c) as g:
        g.initialize()
        g.run_op("UPDATE_BUCKETS")
        n = [C.c_longlong(), C.c_longlong()]
        mps.lib().mpsgpu_launch_count(C.byref(n[0]))
        g.run_op("VISCOSITY")
        mps.lib().mpsgpu_launch_count(C.byref(n[1]))
        assert n[1].value - n[0].value == launches
