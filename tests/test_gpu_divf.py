"""The FP32 quotient of two float-float values is the FP64 quotient rounded to FP32, bit for bit:
random values over FP32's range, quotients at ties of the rounding and within 2^-26 to 2^-48 of them,
powers of two, and zeros, infinities and NaN.
"""
import ctypes as C
import subprocess

import numpy as np
import pytest

from polymps_gb300 import build

pytestmark = pytest.mark.gpu

SRC = """
#include "mps_df.cuh"
__global__ void k(const float2* a, const float2* b, float* y, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = divF(df{a[i].x, a[i].y}, df{b[i].x, b[i].y});
}
extern "C" int run(const float* a, const float* b, float* y, int n) {
    float2 *da, *db;
    float* dy;
    if (cudaMalloc(&da, 8ull * n) || cudaMalloc(&db, 8ull * n) || cudaMalloc(&dy, 4ull * n)) return 1;
    cudaMemcpy(da, a, 8ull * n, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, 8ull * n, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(da, db, dy, n);
    int e = cudaMemcpy(y, dy, 4ull * n, cudaMemcpyDeviceToHost);
    cudaFree(da); cudaFree(db); cudaFree(dy);
    return e;
}
"""


def _split(x):
    h = x.astype(np.float32)
    with np.errstate(invalid="ignore"):
        l = np.where(np.isfinite(h), x - h.astype(np.float64), 0.0).astype(np.float32)
    return np.ascontiguousarray(np.stack([h, l], axis=-1))


def _pairs():
    rng = np.random.default_rng(6)
    n = 1 << 18
    sign = rng.choice([-1.0, 1.0], n)
    for e in (20, 60, 120):
        yield sign * rng.uniform(1, 2, n) * 2.0 ** rng.integers(-e, e, n), rng.uniform(1, 2, n) * 2.0 ** rng.integers(-e, e, n)
    b = rng.uniform(1, 2, n)
    tie = rng.uniform(1, 2, n).astype(np.float32).astype(np.float64) + 2.0 ** -24
    for off in [0.0] + [s * 2.0 ** -k for k in range(26, 49) for s in (-1, 1)]:
        yield sign * (tie + off) * b, b
    two = 2.0 ** rng.integers(-20, 20, n)
    yield two * (1 - 2.0 ** -25 * rng.uniform(0.99, 1.01, n)) * b, b
    s = np.array([0.0, 1.0, np.inf, np.nan, 2.0 ** -130, 2.0 ** 120, -3.0])
    yield tuple(v.ravel() for v in np.meshgrid(s, s))


def test_bits_of_the_rounded_fp64_quotient(tmp_path):
    (tmp_path / "d.cu").write_text(SRC)
    subprocess.run([build._nvcc(), *build.GENCODE, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + build.CSRC, str(tmp_path / "d.cu"), "-o", str(tmp_path / "d.so")], check=True)
    lib = C.CDLL(str(tmp_path / "d.so"))
    P = C.POINTER(C.c_float)
    for a, b in _pairs():
        a, b = _split(a), _split(b)
        y = np.empty(len(a), dtype=np.float32)
        assert lib.run(a.ctypes.data_as(P), b.ctypes.data_as(P), y.ctypes.data_as(P), len(a)) == 0
        with np.errstate(all="ignore"):
            want = (a.astype(np.float64).sum(axis=1) / b.astype(np.float64).sum(axis=1)).astype(np.float32)
        assert np.array_equal(y, want, equal_nan=True)
