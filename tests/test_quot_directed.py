"""The grouped FP64 quotients (csrc/quot.cuh) on operands made to be hard to round: dividends whose quotient lies as near
as possible to the midpoint of two neighbours (A 2^k = M B + d, M odd of 54 bits and d a small odd number, by the
inverse of B modulo a power of two), for divisors just below a power of two, where a reciprocal's rounding is
hardest, and for random ones; and dividends of both zeros. Every form, with the device's and with the host's
reciprocal, against IEEE division on the host, bit for bit."""
import ctypes
import random
import subprocess

import numpy as np
import pytest

from atjup_b200 import build

SRC = r"""
#include <cuda_runtime.h>
#include "quot.cuh"
using namespace atjup;
// the reciprocal, and six quotients per pair: alone, by the device's reciprocal, by the host's, in a group of two, by the
// group's common divisor, and in a group of different divisors with their reciprocals
__global__ void form(const double* a, const double* b, const double* r, double* o, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int j = i + 1 < n ? i + 1 : 0;
    const double a2[2] = {a[i], a[j]}, b2[2] = {b[i], b[j]}, r2[2] = {rcp_of(b[i]), rcp_of(b[j])};
    double q[2];
    o[7 * i] = rcp_of(b[i]);
    o[7 * i + 6] = quot1(a[i], b[i]);
    o[7 * i + 1] = quot1_by(a[i], b[i], rcp_of(b[i]));
    o[7 * i + 2] = quot1_by(a[i], b[i], r[i]);
    quots(a2, b2, q);
    o[7 * i + 3] = q[0];
    const double c2[2] = {a[i], 2.0 * a[i]};
    quots_by(c2, b[i], r[i], q);
    o[7 * i + 4] = q[0];
    quots(a2, b2, r2, q);
    o[7 * i + 5] = q[0];
}
extern "C" int forms(const double* a, const double* b, const double* r, double* o, int n) {
    double *d = nullptr, *w = nullptr;
    if (cudaMalloc(&d, 24ull * n) != cudaSuccess || cudaMalloc(&w, 56ull * n) != cudaSuccess) return -1;
    cudaMemcpy(d, a, 8ull * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, 8ull * n, cudaMemcpyHostToDevice);
    cudaMemcpy(d + 2 * n, r, 8ull * n, cudaMemcpyHostToDevice);
    form<<<(n + 127) / 128, 128>>>(d, d + n, d + 2 * n, w, n);
    const int rc = cudaMemcpy(o, w, 56ull * n, cudaMemcpyDeviceToHost) != cudaSuccess;
    cudaFree(d);
    cudaFree(w);
    return rc;
}
"""


def hard_pairs():
    """(A, B): 53-bit integers, A / B next to the midpoint of two 53-bit numbers"""
    rng = random.Random(11)
    near = [2 ** 53 - d for d in range(1, 20001, 2)]
    near += [2 ** 53 - (rng.randrange(1, 2 ** e) | 1) for e in range(15, 49) for _ in range(500)]
    low = [2 ** 52 + (rng.randrange(1, 2 ** 30) | 1) for _ in range(5000)]
    some = [rng.randrange(2 ** 52, 2 ** 53) | 1 for _ in range(30000)]
    for B in near + low + some:
        for k in (53, 54):
            inv = pow(B, -1, 2 ** k)
            for d in (1, -1, 3, -3):
                M = -d * inv % 2 ** k
                if k == 53:
                    M += 2 ** 53
                A = (M * B + d) >> k
                if M >= 2 ** 53 and 2 ** 52 <= A < 2 ** 53:
                    assert A << k == M * B + d and M & 1
                    yield A, B


def test_pairs_are_next_to_midpoints():
    from fractions import Fraction
    n = 0
    for A, B in hard_pairs():
        n += 1
        if n % 997:
            continue
        q = Fraction(A, B) * (2 ** 53 if A >= B else 2 ** 54)      # 54 bits: odd halves are the midpoints
        m = round(q)
        assert m % 2 == 1 and 0 < abs(q - m) <= Fraction(3, B)
    assert n > 60000


@pytest.mark.gpu
def test_hard_quotients_equal_division(tmp_path):
    src, so = tmp_path / "q.cu", tmp_path / "q.so"
    src.write_text(SRC)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I",
                    str(build.CSRC), "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    pairs = np.array(list(hard_pairs()), dtype=np.float64)
    rng = np.random.default_rng(1)
    a, b = (np.ldexp(pairs[:, q], rng.integers(-300, 200, len(pairs))) for q in (0, 1))
    a, b = a * rng.choice([-1.0, 1.0], len(a)), b * rng.choice([-1.0, 1.0], len(b))
    z = np.array([0.0, -0.0, 0.0, -0.0])                            # both zeros over both signs
    a, b = np.concatenate([a, z]), np.concatenate([b, [3.0, 3.0, -7.0, -7.0]])
    r, o = 1.0 / b, np.empty((len(a), 7))
    ptr = lambda x: x.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    lib.forms.argtypes = [ctypes.POINTER(ctypes.c_double)] * 4 + [ctypes.c_int]
    assert lib.forms(ptr(a), ptr(b), ptr(r), ptr(o), len(a)) == 0
    want = np.column_stack([r] + [a / b] * 6)
    bad = o.view(np.uint64) != want.view(np.uint64)
    bad[b < 0, 0] = False                       # the reciprocal is for positive divisors
    where = np.nonzero(bad.any(axis=1))[0][:5]
    assert not bad.any(), f"{bad.sum(axis=0)} of {len(a)}, first {[(a[i].hex(), b[i].hex()) for i in where]}"
