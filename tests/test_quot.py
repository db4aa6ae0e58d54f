"""The grouped FP64 quotients (csrc/quot.cuh) against the device's IEEE division: the header compiled into a
small kernel, random operands over the accepted exponents, with divisors near the ends of a binade."""
import ctypes
import subprocess

import pytest

from atjup_b200 import build

pytestmark = pytest.mark.gpu

SRC = r"""
#include <cuda_runtime.h>
#include "quot.cuh"
using namespace atjup;
__device__ unsigned long long rng(unsigned long long& s) { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
__global__ void check(unsigned long long* bad) {
    unsigned long long s = 88172645463325252ull ^ ((blockIdx.x * 256ull + threadIdx.x + 1) * 0x9E3779B97F4A7C15ull);
    for (int i = 0; i < 8; i++) rng(s);
    unsigned long long n = 0;
    for (int i = 0; i < 256; i++) {
        double a[3], b[3], o[3];
        for (int u = 0; u < 3; u++) {
            unsigned long long ma = rng(s) & 0xfffffffffffffull, mb = rng(s) & 0xfffffffffffffull;
            if (i % 16 == 0) mb = 0xfffffffffffffull - (rng(s) & 15);
            if (i % 16 == 1) mb = rng(s) & 15;
            const unsigned long long ea = 1023 + (int)(rng(s) % 801) - 400, eb = 1023 + (int)(rng(s) % 801) - 400;
            a[u] = __longlong_as_double((ea << 52) | ma | (rng(s) << 63));
            b[u] = __longlong_as_double((eb << 52) | mb | (rng(s) << 63));
            if (i == 5) a[u] = 0.0;
            if (i == 6) b[u] = 0.0;                  // the group's plain divisions
            if (i == 7) a[u] = __longlong_as_double(0x7ff0000000000000ll);
            if (i == 8) a[u] = 4.9e-324;
        }
        quots(a, b, o);
        for (int u = 0; u < 3; u++) {
            const double w = a[u] / b[u], x = quot1(a[u], b[u]);
            n += !(o[u] == w || (o[u] != o[u] && w != w));
            n += !(x == w || (x != x && w != w));
        }
    }
    atomicAdd(bad, n);
}
extern "C" long long mismatches() {
    unsigned long long* d = nullptr; unsigned long long h = ~0ull;
    if (cudaMalloc(&d, 8) != cudaSuccess) return -1;
    cudaMemset(d, 0, 8);
    check<<<512, 256>>>(d);
    if (cudaMemcpy(&h, d, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    cudaFree(d);
    return (long long)h;
}
"""


def test_quotients_equal_division(tmp_path):
    src, so = tmp_path / "q.cu", tmp_path / "q.so"
    src.write_text(SRC)
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I",
                    str(build.CSRC), "-o", str(so), str(src)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.mismatches.restype = ctypes.c_longlong
    assert lib.mismatches() == 0
