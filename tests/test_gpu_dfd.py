"""The split of an FP64 value into two floats: h = fl32(x) and l = fl32(x - h), as NumPy rounds them,
bit for bit (the sign of a zero l aside): random significands over FP32's range, ties and their
neighbours at every last bit, significands that round up into the next binade, and the values on
either side of the range of the integer form.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from polymps_gb300 import build

pytestmark = pytest.mark.gpu

SRC = """
#include "mps_df.cuh"
__global__ void k(const double* a, float2* y, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) { const df v = dfD(a[i]); y[i] = make_float2(v.h, v.l); }
}
extern "C" int run(const double* a, float* y, int n) {
    double* da; float2* dy;
    if (cudaMalloc(&da, 8ull * n) || cudaMalloc(&dy, 8ull * n)) return 1;
    cudaMemcpy(da, a, 8ull * n, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(da, dy, n);
    int e = cudaMemcpy(y, dy, 8ull * n, cudaMemcpyDeviceToHost);
    cudaFree(da); cudaFree(dy);
    return e;
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("dfd")
    (d / "s.cu").write_text(SRC)
    subprocess.run([build._nvcc(), *build.GENCODE, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + build.CSRC, str(d / "s.cu"), "-o", str(d / "s.so")], check=True)
    lib = C.CDLL(str(d / "s.so"))

    def run(a):
        a = np.ascontiguousarray(a, dtype=np.float64)
        y = np.empty((len(a), 2), dtype=np.float32)
        assert lib.run(a.ctypes.data_as(C.POINTER(C.c_double)), y.ctypes.data_as(C.POINTER(C.c_float)),
                       C.c_int(len(a))) == 0
        return y
    return run


def _values():
    rng = np.random.default_rng(2)
    frac = rng.integers(0, 1 << 52, 1 << 20, dtype=np.int64)
    low = np.array([0, 1, (1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1, (1 << 24) + 1, (1 << 28) + (1 << 23) + 3])
    edge = ((rng.integers(0, 1 << 23, (4096, 1)) << 29) + low).ravel()
    edge = np.concatenate([edge, (((1 << 23) - 1) << 29) + low, low])
    frac = np.concatenate([frac, edge])
    for lo, hi in ((926, 1150), (926, 927), (1149, 1150), (880, 926)):
        e = rng.integers(lo, hi, len(frac), dtype=np.int64)
        sign = rng.integers(0, 2, len(frac), dtype=np.int64) << 63
        yield ((e << 52) | frac | sign).view(np.float64)
    yield np.array([0.0, -0.0, 1e-300, -1e-300, 3e38, -3e38, 1.0, -1.0])


def test_split_is_correctly_rounded(split):
    for a in _values():
        y = split(a)
        h = a.astype(np.float32)
        l = (a - h.astype(np.float64)).astype(np.float32)
        assert np.array_equal(y[:, 0], h) and np.array_equal(y[:, 1], l)


def test_not_finite(split):
    y = split(np.array([np.inf, -np.inf, np.nan, 1e300]))
    assert y[0, 0] == np.inf and y[1, 0] == -np.inf and np.isnan(y[2, 0]) and y[3, 0] == np.inf
