"""Network calls on host arrays: features read in place (16-byte aligned arrays) and copied first
(any other alignment) give the same outputs, at the edges of the 128-row tiles and past the
workspace that is kept between calls; a larger call after a smaller one and back.

Outputs are compared bit for bit (the same kernel on the same values).  The gradient sums its
blocks' parts in the order they arrive, so two runs differ by the rounding of at most 1,024
FP32 additions per entry: 1e-4 of the largest entry.
"""
import numpy as np
import pytest

from polymps_gb300 import abi, cases

pytestmark = pytest.mark.gpu


def _place(a, offset):
    """A copy of a at `offset` floats from a 64-byte boundary."""
    raw = np.zeros(a.size + 32, np.float32)
    start = (-raw.ctypes.data // 4) % 16 + offset
    v = raw[start:start + a.size].reshape(a.shape)
    v[...] = a
    return v


@pytest.fixture(scope="module")
def net(mps_lib):
    from polymps_gb300 import mps
    rng = np.random.default_rng(4)
    g = mps.MpsGpu(cases.config(3, scale=8.0))
    norm = np.concatenate([np.zeros(16), np.ones(16), [0.0, 1.0]]).astype(np.float32)
    g.mlp_set_weights((0.2 * rng.standard_normal(abi.MLP_NPARAM)).astype(np.float32), norm)
    yield g
    g.close()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 70001, 64])
def test_forward_alignment(net, n):
    f = np.random.default_rng(n).standard_normal((n, abi.MLP_NFEAT)).astype(np.float32)
    a, b = net.mlp_forward(_place(f, 0)), net.mlp_forward(_place(f, 1))
    assert np.any(a) and np.array_equal(a, b)


@pytest.mark.parametrize("n", [1, 129, 70001])
def test_forward_output_in_the_features_memory(net, n):
    from polymps_gb300 import mps
    f = np.random.default_rng(n).standard_normal((n, abi.MLP_NFEAT)).astype(np.float32)
    want = net.mlp_forward(f)
    for first in (0, (abi.MLP_NFEAT - 1) * n):   # the outputs over the first or the last n features
        buf = _place(f, 0).reshape(-1)
        out = buf[first:first + n]
        assert mps.lib().mpsgpu_mlp_forward(net.h, abi.fptr(buf), n, abi.fptr(out)) == 0
        assert np.array_equal(out, want)


@pytest.mark.parametrize("n", [64, 128, 65536 + 64, 2097152, 64])
def test_gradient_alignment(net, n):
    rng = np.random.default_rng(n)
    f = rng.standard_normal((n, abi.MLP_NFEAT)).astype(np.float32)
    t = rng.standard_normal(n).astype(np.float32)
    (ga, la), (gb, lb) = net.mlp_gradient(_place(f, 0), t), net.mlp_gradient(_place(f, 1), t)
    assert np.any(ga) and np.abs(ga - gb).max() <= 1e-4 * np.abs(ga).max()
    assert abs(la - lb) <= 1e-4 * abs(la)
