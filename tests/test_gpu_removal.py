"""Removal of fluid particles outside the domain where the grid strides over the particles (more
than 608 blocks of 256): particles pushed out at the first, the last and at block and round edges,
against the reference's serial loop (src/MpsParticle.cpp, swap with the last live index, which is
not looked at again) restated on the host.  Whole arrays are moved, so the comparison is exact.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu

ROUND = 608 * 256


@pytest.mark.parametrize("cells", [(38, 64, 64), (40, 64, 65), (71, 67, 33)])   # one round exactly, two, a ragged two
def test_removal_over_rounds(mps_lib, cells):
    from polymps_gb300 import mps
    l0 = 0.01
    size = tuple(l0 * k for k in cells)
    c = cases.dam3d_polygon(l0=l0, fluid=size, tank=(2.683 * size[0], size[1], 2.0 * size[2]), mode="wc", dt=1e-4)
    n = len(c.pos)
    assert n == cells[0] * cells[1] * cells[2]
    g = mps.MpsGpu(c)
    g.initialize()
    g.run_op("UPDATE_BUCKETS")
    pos = g.get(abi.F_POS)
    press = np.arange(n, dtype=np.float64)
    xout = g.params.domainMax[0] - 0.5 * g.params.bucketSide
    out = sorted({0, 255, 256, n // 2, ROUND - 1, n - 2, n - 1} | ({ROUND} if n > ROUND else set()))
    pos[out, 0] = xout
    g.set(abi.F_POS, pos)
    g.set(abi.F_PRESS, press)
    for _ in range(2):   # the second call finds those copied into freed places; its counters start at zero
        order = list(range(len(pos)))
        live, r = len(order), 0
        gone = pos[:, 0] == xout
        while r < live:
            if gone[r]:
                order[r] = order[live - 1]
                live -= 1
            r += 1
        g.run_op("OUT_OF_DOMAIN")
        assert g.n == live
        order = order[:live]
        pos, press = pos[order], press[order]
        assert np.array_equal(g.get(abi.F_POS)[:live], pos)
        assert np.array_equal(g.get(abi.F_PRESS)[:live], press)
    g.close()
