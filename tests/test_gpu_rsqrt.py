"""The FP64 reciprocal square root of the pair weights (one Halley step from the FP32 estimate)
against 1 / sqrt in extended precision: random arguments over the FP32 range, arguments around
the powers of two where the estimate lies at the edge of a binade, and the arguments left to
rsqrt().

Bound: half an ulp for the last multiply-add, the series' remainder 5/16 e^3 < 2^-62 and the
factor's 2^-41 times e < 2^-20, together below 0.51 ulp.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from polymps_gb300 import build

pytestmark = pytest.mark.gpu

SRC = """
#include "mps_common.cuh"
__global__ void k(const double* a, double* y, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = rsqrtHalley(a[i]);
}
extern "C" int run(const double* a, double* y, int n) {
    double *da, *dy;
    if (cudaMalloc(&da, 8ull * n) || cudaMalloc(&dy, 8ull * n)) return 1;
    cudaMemcpy(da, a, 8ull * n, cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(da, dy, n);
    int e = cudaMemcpy(y, dy, 8ull * n, cudaMemcpyDeviceToHost);
    cudaFree(da); cudaFree(dy);
    return e;
}
"""


@pytest.fixture(scope="module")
def rsqrt(tmp_path_factory):
    d = tmp_path_factory.mktemp("rsqrt")
    (d / "r.cu").write_text(SRC)
    subprocess.run([build._nvcc(), *build.GENCODE, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + build.CSRC, "-I" + os.path.join(build.PKG, "csrc"), str(d / "r.cu"), "-o", str(d / "r.so")],
                   check=True)
    lib = C.CDLL(str(d / "r.so"))

    def run(a):
        a = np.ascontiguousarray(a, dtype=np.float64)
        y = np.empty_like(a)
        P = C.POINTER(C.c_double)
        assert lib.run(a.ctypes.data_as(P), y.ctypes.data_as(P), C.c_int(len(a))) == 0
        return y
    return run


def _ulps(a, y):
    exact = 1 / np.sqrt(a.astype(np.longdouble))
    return np.abs((y.astype(np.longdouble) - exact) / np.spacing(y).astype(np.longdouble))


def test_random_arguments(rsqrt):
    rng = np.random.default_rng(1)
    a = rng.uniform(1.0, 4.0, 1 << 20) * 2.0 ** rng.integers(-125, 125, 1 << 20)
    assert _ulps(a, rsqrt(a)).max() <= 0.51


def test_binade_edges(rsqrt):
    base = 4.0 ** np.arange(-60, 60)
    rel = np.concatenate([k * 2.0 ** -np.arange(18, 53) for k in (-3.0, -1.0, 1.0, 3.0)] + [[0.0]])
    a = (base[:, None] * (1.0 + rel)).ravel()
    a = np.concatenate([a, 2.0 * a])
    assert _ulps(a, rsqrt(a)).max() <= 0.51


def test_outside_the_fp32_range(rsqrt):
    lo, hi = 2.0 ** -126, 2.0 ** 128
    a = np.array([lo, np.nextafter(lo, 0), np.nextafter(hi, 0), hi, 1e-300, 1e300, 5e-324, 2.0 ** -130, 2.0 ** 130])
    assert _ulps(a, rsqrt(a)).max() <= 1.0
    y = rsqrt(np.array([0.0, np.inf, -1.0, np.nan]))
    assert y[0] == np.inf and y[1] == 0.0 and np.isnan(y[2]) and np.isnan(y[3])
