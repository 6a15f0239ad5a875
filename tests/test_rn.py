"""The branch-free square root and quotients of csrc/pd_rn.cuh are IEEE's, bit
for bit: on random operands, on the operands next to which a square root or
quotient lies closest to a rounding boundary (built here by number theory),
and on divisors next to a power of two."""
import ctypes as C
import math
import os
import random
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = r"""
#include <cstdint>
#include "pd_rn.cuh"
__global__ void k(const double* a, const double* b, double* s, double* q, unsigned char* ok, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double r, y;
    pd::rn_sqrt_rcp(b[i], r, y);
    s[i] = r;
    q[i] = pd::rn_div_signed(a[i], r, y);
    ok[i] = (pd::rn_range(b[i]) ? 1 : 0) | (pd::rn_quotient_ok(a[i]) ? 2 : 0);
}
extern "C" int rn_run(const double* a, const double* b, double* s, double* q, unsigned char* ok, int n) {
    double* d[4];
    unsigned char* f;
    for (int v = 0; v < 4; ++v) cudaMalloc(&d[v], n * sizeof(double));
    cudaMalloc(&f, n);
    cudaMemcpy(d[0], a, n * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(d[1], b, n * sizeof(double), cudaMemcpyHostToDevice);
    k<<<(n + 255) / 256, 256>>>(d[0], d[1], d[2], d[3], f, n);
    cudaMemcpy(s, d[2], n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaMemcpy(q, d[3], n * sizeof(double), cudaMemcpyDeviceToHost);
    cudaMemcpy(ok, f, n, cudaMemcpyDeviceToHost);
    for (int v = 0; v < 4; ++v) cudaFree(d[v]);
    cudaFree(f);
    return (int)cudaGetLastError();
}
"""


def roots_of(j, bits):
    """Odd M with M^2 = j modulo 2^bits (j = 1 modulo 8): four of them."""
    x = 1
    for k in range(3, bits):
        if (x * x - j) >> k & 1:
            x += 1 << (k - 1)
    mod = 1 << bits
    assert (x * x - j) % mod == 0
    return {v % mod for v in (x, -x, x + mod // 2, -x + mod // 2)}


def hard_squares():
    """Every a in [1, 4) within 511 * 2^-106 of the square of a midpoint m =
    M 2^-53 of two doubles in [1, 2)."""
    out = set()
    for j in range(-511, 512):
        if j % 8 != 1:
            continue
        for bits, lo, hi in ((54, 1 << 53, math.isqrt(1 << 107)), (55, math.isqrt(1 << 107) + 1, 1 << 54)):
            for M in roots_of(j % (1 << bits), bits):
                for k in range(0, 2):
                    m = M + (k << bits) if bits == 54 else M
                    if lo <= m < hi:
                        a = m * m - j
                        assert a % (1 << bits) == 0
                        out.add(float(a >> bits) * 2.0 ** (bits - 106))
    return sorted(out)


def hard_quotients(rng):
    """(a, b) with a / b closer to a midpoint than 4 * 2^-105: b random and
    the largest mantissas."""
    out = []
    divisors = [rng.randrange(1 << 52, 1 << 53) | 1 for _ in range(4000)]
    divisors += [(1 << 53) - 1 - 2 * k for k in range(200)] + [(1 << 52) + 1 + 2 * k for k in range(50)]
    for B in divisors:
        inv = pow(B, -1, 1 << 53)
        for k in (-3, -2, -1, 1, 2, 3):
            M = (1 << 53) + (-k * inv) % (1 << 53)  # B M = -k modulo 2^53
            A, rest = divmod(B * M + k, 1 << 53)
            assert rest == 0
            if M & 1 and (A < 1 << 53 or not A & 1):
                out.append((float(A), float(B)))
    return out


def test_hard_operands_lie_where_they_should():
    a = hard_squares()
    assert len(a) > 120
    for v in a[:50]:
        n = int(v * 2 ** 60) << 46  # v 2^106
        m = math.isqrt(n)
        assert min(abs(n - x * x) for x in (m, m + 1) if x & 1) <= 511
    q = hard_quotients(random.Random(1))
    assert len(q) > 3000


@pytest.mark.gpu
def test_square_roots_and_quotients_are_ieee(tmp_path):
    cu, so = tmp_path / "rn.cu", tmp_path / "rn.so"
    cu.write_text(SRC)
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-gencode", "arch=compute_100a,code=sm_100a",
                    "-O3", "-std=c++17", "-fmad=false", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + os.path.join(ROOT, "pdmtel_b200", "csrc"), str(cu), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    rng = random.Random(7)
    g = np.random.default_rng(7)
    a, b = [], []
    for v in hard_squares():
        for e in (-398, -20, 0, 42, 396):
            b.append(v * 2.0 ** e)
            a.append(rng.uniform(-2, 2))
    for x, y in hard_quotients(rng):
        for e in (-390, 0, 250):
            a.append(x * 2.0 ** e)
            b.append((y * y) * 2.0 ** 60)  # its root is y 2^30: the square of a double has that root
    n = 2_000_000
    b = np.concatenate([b, np.exp2(g.uniform(-399, 399, n)) * g.uniform(1, 2, n) / 2])
    a = np.concatenate([a, g.choice([-1, 1], n) * np.exp2(g.uniform(-499, 498, n))])
    a = np.concatenate([a, [0.0, -0.0, 5e-324, -1e-310, 1e-300, np.inf, np.nan, 1e200]])
    b = np.concatenate([b, [2.0] * 8])
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    s, q, ok = np.empty_like(a), np.empty_like(a), np.empty(a.size, np.uint8)
    p = lambda v: v.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert lib.rn_run(p(a), p(b), p(s), p(q), p(ok), C.c_int(a.size)) == 0
    assert np.array_equal(s, np.sqrt(b))
    assert np.all(ok & 1)
    inside = (ok & 2) != 0
    assert np.array_equal(inside[-8:], [True, True, False, False, False, False, False, False])
    assert np.all(inside[:-8])
    want = a[inside] / np.sqrt(b[inside])
    assert np.array_equal(q[inside].view(np.int64), want.view(np.int64))
