"""The correction matrix that the PND sweep leaves in staging arrays for the matrix operator to
publish: what is published is the matrix of the current state in either tier.  Against the FP64 CPU
oracle running the same operators: 1e-10 normwise in the FP64 tier, 1e-8 in the float-float one.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

from test_gpu_parity import relerr, step_ops, sync

pytestmark = pytest.mark.gpu


def _pair(oracle_mod, mps, precision, **kw):
    c = cases.dam3d_polygon(l0=0.01, fluid=(0.12, 0.11, 0.13), tank=(0.4, 0.11, 0.4), jitter=0.03, **kw)
    o = oracle_mod.Oracle(c)
    o.set_solver(1e-12)
    g = mps.MpsGpu(c, tol=1e-12, precision=precision)
    o.initialize()
    g.initialize()
    return o, g


def test_float_float_matrix_across_tiers(oracle_mod, mps_lib):
    """The FP64 tier's operators leave the float-float copy of the matrix alone."""
    from polymps_gb300 import mps
    o, g = _pair(oracle_mod, mps, abi.PRECISION_DF32)
    sync(o, g)
    ops = step_ops(o.params)
    for op in ops[: ops.index("CORRECTION_MATRIX") + 1]:
        o.run_op(op)
        g.run_op(op)
    g.set_precision(abi.PRECISION_FP64)
    for op in ("PND_NEIGH_NPCD", "CORRECTION_MATRIX"):
        o.run_op(op)
        g.run_op(op)
    for f in (abi.F_CORR1, abi.F_CORR2, abi.F_CORR3):
        assert relerr(g.get(f), o.get(f)) <= 1e-10
    g.set_precision(abi.PRECISION_DF32)
    # the same pressures on both sides, without the field interface (it would copy the matrix)
    o.set(abi.F_PRESS, g.get(abi.F_PRESS))
    o.run_op("PRESS_GRADIENT")
    g.run_op("PRESS_GRADIENT")
    assert np.any(o.get(abi.F_ACC))
    assert relerr(g.get(abi.F_ACC), o.get(abi.F_ACC)) <= 1e-8
    g.close()
    o.close()


@pytest.mark.parametrize("alone", [True, False])
def test_fp64_matrix_of_its_own_operator_and_of_a_step(oracle_mod, mps_lib, alone):
    """The FP64 PND operator called alone leaves the matrix to the matrix operator; a step forms both
    in one sweep.  The published matrix is the oracle's either way."""
    import ctypes as C
    from polymps_gb300 import mps
    o, g = _pair(oracle_mod, mps, abi.PRECISION_FP64)
    sync(o, g)
    if alone:
        ops = step_ops(o.params)
        for op in ops[: ops.index("CORRECTION_MATRIX")]:
            o.run_op(op)
            g.run_op(op)
        n = [C.c_longlong(), C.c_longlong()]
        mps.lib().mpsgpu_launch_count(C.byref(n[0]))
        o.run_op("CORRECTION_MATRIX")
        g.run_op("CORRECTION_MATRIX")
        mps.lib().mpsgpu_launch_count(C.byref(n[1]))
        assert n[1].value - n[0].value == 1   # 0: published from what the PND sweep formed
    else:
        o.step()
        g.step()
    for f in (abi.F_CORR1, abi.F_CORR2, abi.F_CORR3):
        assert relerr(g.get(f), o.get(f)) <= 1e-10
    g.close()
    o.close()


def test_matrix_of_the_fp64_tier_in_the_float_float_one(oracle_mod, mps_lib):
    """A float-float pressure gradient after a change of tier reads the matrix the FP64 one formed."""
    from polymps_gb300 import mps
    o, g = _pair(oracle_mod, mps, abi.PRECISION_FP64)
    sync(o, g)
    ops = step_ops(o.params)
    for op in ops[: ops.index("CORRECTION_MATRIX") + 1]:
        o.run_op(op)
        g.run_op(op)
    g.set_precision(abi.PRECISION_DF32)
    # the same pressures on both sides, without the field interface (it would copy the matrix)
    o.set(abi.F_PRESS, g.get(abi.F_PRESS))
    o.run_op("PRESS_GRADIENT")
    g.run_op("PRESS_GRADIENT")
    assert np.any(o.get(abi.F_ACC))
    assert relerr(g.get(abi.F_ACC), o.get(abi.F_ACC)) <= 1e-8
    g.close()
    o.close()
