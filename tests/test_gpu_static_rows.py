"""mpsgpu_pcg_solve_static at the edges of its row split: systems of one row up to the limit,
around the rows of a block and of a round, with rows of 1 to about 70 entries in no order and
a diagonal at any place, against a dense solve or (the limit) a system with a known solution.
The matrices are symmetric with 4 |off-diagonal row sum| <= diagonal, so their condition
number after the Jacobi scaling is below 2 and a solve to 1e-12 is within 1e-11 of the
solution; the bound asked for is 1e-10.
"""
import ctypes as C

import numpy as np
import pytest

from polymps_gb300 import abi

pytestmark = pytest.mark.gpu


def _system(n, most, seed):
    rng = np.random.default_rng(seed)
    a = {}
    for i in range(n):
        for j in rng.integers(0, n, size=rng.integers(0, most // 2 + 1)):
            if i != j:
                a[(i, int(j))] = a[(int(j), i)] = -rng.uniform(0.1, 1.0)
    rows = [[] for _ in range(n)]
    for (i, j), v in a.items():
        rows[i].append((j, v))
    dense = np.zeros((n, n)) if n <= 4000 else None
    ptr, col, val = [0], [], []
    for i, r in enumerate(rows):
        r.append((i, 4.0 * sum(-v for _, v in r) + rng.uniform(0.5, 2.0)))
        rng.shuffle(r)
        for j, v in r:
            j = int(j)
            col.append(j), val.append(v)
            if dense is not None:
                dense[i, j] = v
        ptr.append(len(col))
    return np.array(ptr, np.int32), np.array(col, np.int32), np.array(val), dense


@pytest.mark.parametrize("n,most", [(1, 0), (2, 2), (3, 4), (31, 70), (63, 20), (64, 20), (65, 70), (129, 3), (1000, 40),
                                    (2047, 66), (3001, 30), (abi.STATIC_MAX_ROWS, 2), (abi.STATIC_MAX_ROWS - 37, 0)])
def test_static_solver_row_split(mps_lib, n, most):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    if n > 4000:   # diagonal, or diagonal with one coupling per pair of distant rows
        i = np.arange(n)
        partner = n - 1 - i
        ptr = (np.arange(n + 1) * (2 if most else 1)).astype(np.int32)
        col = (np.stack([partner, i], 1).ravel() if most else i).astype(np.int32)
        val = np.stack([np.full(n, -1.0), np.full(n, 4.5)], 1).ravel() if most else rng.uniform(1, 2, n)
        x = rng.normal(size=n)
        b = 4.5 * x - x[partner] if most else val * x
    else:
        ptr, col, val, dense = _system(n, most, n)
        b = rng.normal(size=n)
        x = np.linalg.solve(dense, b)
    dev = [torch.from_numpy(a).cuda() for a in (ptr, col, val, b)]
    got = []
    for _ in range(2):
        y = torch.zeros(n, dtype=torch.float64, device="cuda")
        it, res = C.c_int(), C.c_double()
        rc = mps_lib.mpsgpu_pcg_solve_static(n, *[t.data_ptr() for t in dev], y.data_ptr(), 1e-12, 1000,
                                             torch.cuda.current_stream().cuda_stream, C.byref(it), C.byref(res))
        assert rc == 0, mps_lib.mpsgpu_pcg_static_error()
        assert res.value <= 1.1e-12
        got.append(y.cpu().numpy())
    assert np.array_equal(got[0], got[1])
    assert np.linalg.norm(got[0] - x) <= 1e-10 * np.linalg.norm(x)
