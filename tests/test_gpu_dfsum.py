"""The float-float accumulators of the pair sums: 128 positive terms (a full neighbour row) of
products and of single values, against extended precision.

A step of a normalised sum rounds its low part twice, each time by at most 2^-49 of the partial sum s_k,
uniformly: an rms of 2^-49 sqrt(2 / 3) s_k.  With s_k growing linearly the errors of n steps add up to
2^-49 sqrt(2 n) / 3 of the total, 2^-46.6 for 128 terms, and the mean magnitude is below the rms.
"""
import ctypes as C
import subprocess

import numpy as np
import pytest

from polymps_gb300 import build

pytestmark = pytest.mark.gpu

TERMS, ROWS = 128, 1 << 13
SRC = """
#include "mps_df.cuh"
__global__ void k(const float2* a, const float2* b, float2* y, int rows, int terms, int products) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows) return;
    df s = dfF(0.f);
    for (int t = 0; t < terms; t++) {
        const float2 u = a[t * rows + i], v = b[t * rows + i];
        if (products) mac(s, df{u.x, u.y}, df{v.x, v.y});
        else acc(s, df{u.x, u.y});
    }
    y[i] = make_float2(s.h, s.l);
}
extern "C" int run(const float* a, const float* b, float* y, int rows, int terms, int products) {
    float2 *da, *db, *dy;
    const size_t n = 8ull * rows * terms;
    if (cudaMalloc(&da, n) || cudaMalloc(&db, n) || cudaMalloc(&dy, 8ull * rows)) return 1;
    cudaMemcpy(da, a, n, cudaMemcpyHostToDevice);
    cudaMemcpy(db, b, n, cudaMemcpyHostToDevice);
    k<<<(rows + 127) / 128, 128>>>(da, db, dy, rows, terms, products);
    int e = cudaMemcpy(y, dy, 8ull * rows, cudaMemcpyDeviceToHost);
    cudaFree(da); cudaFree(db); cudaFree(dy);
    return e;
}
"""


def _split(x):
    h = x.astype(np.float32)
    return np.stack([h, (x - h.astype(np.float64)).astype(np.float32)], axis=-1)


def _value(p):
    return p[..., 0].astype(np.longdouble) + p[..., 1].astype(np.longdouble)


@pytest.mark.parametrize("products", [1, 0])
def test_mean_error_of_a_full_row(tmp_path, products):
    (tmp_path / "m.cu").write_text(SRC)
    subprocess.run([build._nvcc(), *build.GENCODE, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + build.CSRC, str(tmp_path / "m.cu"), "-o", str(tmp_path / "m.so")], check=True)
    lib = C.CDLL(str(tmp_path / "m.so"))
    rng = np.random.default_rng(4)
    a = _split(rng.uniform(0, 1, (TERMS, ROWS)))
    b = _split(rng.uniform(1, 2, (TERMS, ROWS)))
    y = np.empty((ROWS, 2), dtype=np.float32)
    P = C.POINTER(C.c_float)
    assert lib.run(a.ctypes.data_as(P), b.ctypes.data_as(P), y.ctypes.data_as(P), ROWS, TERMS, products) == 0
    exact = (_value(a) * _value(b) if products else _value(a)).sum(axis=0)
    err = np.abs((_value(y) - exact) / exact)
    assert float(err.mean()) <= 2.0 ** -46.6
