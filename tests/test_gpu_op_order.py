"""Operators called in another order than a step's work on the current state: the start-of-step
sweeps after the particles have moved without a bucket build in between, and after an operator
that refreshes only some of the FP32 position copies (the list filter, the dummy velocities).
Particles move by up to 0.6 l0, four times the skin of the start-of-step list.

Both sides run the same operators from one state, against the FP64 CPU oracle: sums of at most 128
terms, so 1e-10 normwise in the FP64 tier and 1e-8 in the float-float one, times ten for the
operators before that move the particles.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

from test_gpu_parity import relerr, sync

pytestmark = pytest.mark.gpu

FILTERED = ["UPDATE_BUCKETS", "VISCOSITY", "ADD_GRAVITY", "PREDICT", "COLLISION"]
ORDERS = {
    "viscosity_after_filter": FILTERED + ["VISCOSITY"],
    "gradient_after_filter": FILTERED + ["PREDICT_PRESS_GRADIENT"],
    "viscosity_after_move": ["UPDATE_BUCKETS", "PREDICT", "VISCOSITY"],
    "gradient_after_move": ["UPDATE_BUCKETS", "VISCOSITY", "PREDICT", "PREDICT_PRESS_GRADIENT"],
    "viscosity_after_dummy": ["UPDATE_BUCKETS", "PREDICT", "DUMMY_VELOCITY", "VISCOSITY"],
    "viscosity_after_shift": ["UPDATE_BUCKETS", "VISCOSITY", "PREDICT", "COLLISION", "CORRECT", "SHIFTING", "VISCOSITY"],
}


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_DF32])
@pytest.mark.parametrize("name", list(ORDERS))
def test_operators_see_the_current_positions(oracle_mod, mps_lib, name, precision):
    from polymps_gb300 import mps
    if "dummy" in name:
        c = cases.dam2d_particle_walls(jitter=0.03)
    else:
        c = cases.dam3d_polygon(l0=0.01, fluid=(0.24, 0.25, 0.21), tank=(0.7, 0.25, 0.6), jitter=0.03,
                                mode="wc" if "shift" in name else "inc")
    c.params.update(relaxPress=0.5)
    o = oracle_mod.Oracle(c)
    o.set_solver(1e-12)
    g = mps.MpsGpu(c, tol=1e-12, precision=precision)
    o.initialize()
    g.initialize()
    rng = np.random.default_rng(5)
    top = 0.6 * c.params["partDist"] / c.params["timeStep"] / np.sqrt(3)
    o.set(abi.F_VEL, rng.uniform(-top, top, (c.n, 3)) * ([1, 1, 0] if c.params["dim"] == 2 else [1, 1, 1]))
    o.set(abi.F_PRESS, 1e3 * rng.uniform(0, 1, c.n))
    o.set_velmax(0.0)   # the GPU has run no corrector yet
    sync(o, g)
    for op in ORDERS[name]:
        o.run_op(op)
        g.run_op(op)
    rtol = 1e-9 if precision == abi.PRECISION_FP64 else 1e-7
    a, b = g.get(abi.F_ACC), o.get(abi.F_ACC)
    assert np.any(b)
    assert relerr(a, b) <= rtol
    g.close()
    o.close()
