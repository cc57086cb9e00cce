"""Network gradient with targets at any byte address, as an array read from a packed file may have
them: the kernel reads aligned host arrays in place, and others from a copy.

The gradient sums its blocks' parts in the order they arrive, so two runs differ by the rounding of
at most 1,024 FP32 additions per entry: 1e-4 of the largest entry.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_targets_at_odd_addresses(mps_lib, offset):
    from polymps_gb300 import mps
    n = 192
    rng = np.random.default_rng(4)
    norm = np.concatenate([np.zeros(16), np.ones(16), [0.0, 1.0]]).astype(np.float32)
    with mps.MpsGpu(cases.config(3, scale=8.0)) as g:
        g.mlp_set_weights((0.2 * rng.standard_normal(abi.MLP_NPARAM)).astype(np.float32), norm)
        f = rng.standard_normal((n, abi.MLP_NFEAT)).astype(np.float32)
        t = rng.standard_normal(n).astype(np.float32)
        raw = np.zeros(4 * n + 8, np.uint8)
        odd = np.ndarray((n,), np.float32, buffer=raw, offset=(-raw.ctypes.data) % 4 + offset)
        odd[:] = t
        assert odd.ctypes.data % 4 == offset
        (ga, la), (gb, lb) = g.mlp_gradient(f, t), g.mlp_gradient(f, odd)
        assert np.any(ga) and np.abs(ga - gb).max() <= 1e-4 * np.abs(ga).max()
        assert abs(la - lb) <= 1e-4 * abs(la)
