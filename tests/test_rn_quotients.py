"""The reciprocal square root and the quotient that csrc/pd_rn.cuh forms from
the hardware's seeds, within half a unit in the last place (and a little), on
random operands and on divisors and operands next to a power of two."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include "pd_rn.cuh"
__global__ void k(const double* a, const double* b, double* y, double* q, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = pd::rsqrt_near(b[i]);
    q[i] = pd::quotient_near(a[i], b[i]);
}
extern "C" int run(const double* a, const double* b, double* y, double* q, int n) {
    double* d[4];
    for (int v = 0; v < 4; ++v) cudaMalloc(&d[v], n * sizeof(double));
    cudaMemcpy(d[0], a, n * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d[1], b, n * sizeof(double), cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(d[0], d[1], d[2], d[3], n);
    cudaMemcpy(y, d[2], n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaMemcpy(q, d[3], n * sizeof(double), cudaMemcpyDeviceToHost);
    for (int v = 0; v < 4; ++v) cudaFree(d[v]);
    return (int)cudaGetLastError();
}
"""


def test_reciprocal_root_and_quotient(tmp_path):
    cu, so = tmp_path / "rn.cu", tmp_path / "rn.so"
    cu.write_text(SRC)
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + os.path.join(ROOT, "pdmtel_b200", "csrc"), str(cu), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    g = np.random.default_rng(3)
    n = 2_000_000
    ulp = 2.0 ** -52
    edge = np.concatenate([1 + ulp * np.arange(2000), 2 - ulp * np.arange(1, 2001)])
    b = np.concatenate([np.exp2(g.integers(-399, 399, n)) * g.uniform(1, 2, n), edge, 2 * edge, edge * 2.0 ** -398])
    a = g.choice([-1, 1], b.size) * np.exp2(g.integers(-99, 99, b.size)) * g.uniform(1, 2, b.size)
    a[-12000:-6000] = edge[g.integers(0, edge.size, 6000)]
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    y, q = np.empty_like(a), np.empty_like(a)
    p = lambda v: v.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert lib.run(p(a), p(b), p(y), p(q), C.c_int(a.size)) == 0
    # references with 64-bit mantissas: 2^-11 of a unit
    for got, exact in ((y, 1 / np.sqrt(b.astype(np.longdouble))), (q, a.astype(np.longdouble) / b)):
        assert np.max(np.abs((got - exact) / np.spacing(np.abs(got)))) <= 0.5 + 2.0 ** -9
