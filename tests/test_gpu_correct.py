"""The corrector's maximum speed (reduced as squares, one root per block) is the largest speed of
the velocities it leaves: particle counts at block edges, particles at rest before the step, the
fastest particle first or last.  Both round the same sum of squares and its root, fused or not:
within 4 units of the last place, 1e-15.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(8, 8, 4), (15, 17, 1), (9, 19, 3), (40, 33, 17)])
@pytest.mark.parametrize("kind", ["rest", "first", "last"])
def test_maximum_speed(mps_lib, cells, kind):
    from polymps_gb300 import mps
    l0 = 0.02
    size = tuple(l0 * k for k in cells)
    c = cases.dam3d_polygon(l0=l0, fluid=size, tank=(2.0 * size[0], size[1], 2.0 * size[2] + 0.2), mode="inc")
    vel = np.random.default_rng(len(c.pos)).normal(scale=0.01, size=c.pos.shape)
    if kind == "rest":
        vel[:] = 0.0
    else:
        vel[0 if kind == "first" else -1] = [0.6, 0.0, 0.8]
    g = mps.MpsGpu(c)
    g.initialize()
    for step in range(2):   # the two steps use the two slots of the maximum
        g.set(abi.F_VEL, vel)
        st = g.step()
        want = np.sqrt((g.get(abi.F_VEL) ** 2).sum(-1)).max()
        assert want > 0 and abs(st.velMax - want) <= 1e-15 * want
    g.close()
