"""The FP64 kernels' reciprocal (rcp64) against correctly rounded division.

The hardware's approximation has 20 fraction bits, of the operand and of the
result: it is off by less than 2^-18, so the cubic step leaves less than
2^-54, an eighth of the distance between FP64 numbers near 1; with the last
rounding's half, one unit in the last place bounds the whole."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from uq_b200 import build

SOURCE = r"""
#include "lbm_device.cuh"
__global__ void k(const double *d, double *r, int n)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) r[t] = uqlbm::rcp64(d[t]);
}
extern "C" __attribute__((visibility("default"))) int reciprocals(const double *d, double *r, int n)
{
    double *p = nullptr, *q = nullptr;
    const size_t b = sizeof(double) * n;
    int e = cudaMalloc(&p, b) || cudaMalloc(&q, b) || cudaMemcpy(p, d, b, cudaMemcpyHostToDevice);
    if (!e) {
        k<<<(n + 255) / 256, 256>>>(p, q, n);
        e = cudaGetLastError() || cudaMemcpy(r, q, b, cudaMemcpyDeviceToHost);
    }
    cudaFree(p);
    cudaFree(q);
    return e;
}
"""


@pytest.mark.gpu
def test_reciprocal_is_within_one_unit_of_division(cuda_device, tmp_path):
    src, so = tmp_path / "rcp.cu", tmp_path / "rcp.so"
    src.write_text(SOURCE)
    subprocess.run([build.nvcc(), "-std=c++17", "-O3", *build.ARCH, "-Xcompiler", "-fPIC", "-shared",
                    "-I" + os.path.join(build.HERE, "csrc"), "-o", str(so), str(src)], check=True)
    rng = np.random.default_rng(9)
    m = rng.uniform(1.0, 2.0, 1 << 20)
    # every binade whose reciprocals are normal, mantissas at both ends, and
    # denominators as faces and relaxations form them: sums of products of
    # smoothness terms from epsilon's fourth power (both of its limits) up, 1 + dt/tau
    e = rng.integers(-1021, 1021, m.size)
    d = [np.ldexp(m, e), np.ldexp(1.0, np.arange(-1021, 1022)), np.ldexp(2.0 - 2.0 ** -52, np.arange(-1022, 1021)),
         10.0 * rng.uniform(1, 2, 1 << 16) * 10.0 ** rng.uniform(-142, 142, 1 << 16),
         1.0 + 10.0 ** rng.uniform(-18, 18, 1 << 16)]
    d = np.concatenate(d + [-d[0]])
    r = np.empty_like(d)
    L = C.CDLL(str(so))
    p = C.POINTER(C.c_double)
    assert L.reciprocals(d.ctypes.data_as(p), r.ctypes.data_as(p), C.c_int(d.size)) == 0
    want = 1.0 / d
    ulps = np.abs(r.view(np.int64) - want.view(np.int64))
    assert ulps.max() <= 1, (ulps.max(), d[ulps.argmax()])
