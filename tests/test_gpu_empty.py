"""A system whose last particle has left the domain: the neighbour lists are empty, and no call on
it reports an error."""
import ctypes as C

import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_DF32])
def test_neighbors_of_an_empty_system(mps_lib, precision):
    from polymps_gb300 import mps
    c = cases.dam3d_polygon(l0=0.01, fluid=(0.05, 0.04, 0.06), tank=(0.3, 0.04, 0.3), mode="wc", dt=1e-4)
    with mps.MpsGpu(c, precision=precision) as g:
        g.initialize()
        # the serial loop does not look again at what it copies into a freed place
        while g.n:
            n, pos = g.n, g.get(abi.F_POS)
            pos[:, 0] = g.params.domainMax[0] - 0.5 * g.params.bucketSide
            g.set(abi.F_POS, pos)
            g.run_op("OUT_OF_DOMAIN")
            assert g.n < n
        counts, rows = np.zeros(1, dtype=np.int32), np.zeros(1, dtype=np.int32)
        for nbr in (None, abi.iptr(rows)):
            assert mps.lib().mpsgpu_get_neighbors(g.h, abi.iptr(counts), nbr, C.c_longlong(0)) == 0
        g.run_op("ADD_GRAVITY")
