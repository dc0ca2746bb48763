"""Rounded reciprocals, square roots and quotients without the operators' tests
(csrc/mh_round.cuh, csrc/mh_div.h) against the operators on the GPU.

Every significand, at exponents over the stated range 2^-80 .. 2^80 (both parities
for the square root, the ends of the range, 1), and quotients by such reciprocals
over the ranges in which the denoisers take them: dividends within 2^-60 .. 2^60,
divisors from 1 to 2^30.  The same bits everywhere.
"""
import ctypes as C
import os
import subprocess

import pytest

from meshhashing_gb300 import build as B

pytestmark = pytest.mark.gpu

SRC = r'''
#include "mh_round.cuh"
struct Result { unsigned long long wrong; float a, b; };
__device__ void note(Result *r, float a, float b, float got, float want) {
  if (__float_as_uint(got) == __float_as_uint(want)) return;
  if (atomicAdd(&r->wrong, 1ull) == 0ull) r->a = a, r->b = b;
}
__device__ unsigned mix(unsigned x) {
  x ^= x >> 16, x *= 0x7feb352du, x ^= x >> 15, x *= 0x846ca68bu;
  return x ^ x >> 16;
}
// a float of significand s (23 bits) and exponent e
__device__ float make(unsigned s, int e) { return __uint_as_float((unsigned)(e + 127) << 23 | s); }
__global__ void k_unary(Result *r, int root, int e) {
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < 1u << 23; s += gridDim.x * blockDim.x) {
    const float x = make(s, e);
    note(r, x, 0.0f, root ? sqrt_round(x) : rcp_round(x), root ? sqrtf(x) : 1.0f / x);
  }
}
__global__ void k_quotient(Result *r, int e, unsigned seed) {
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < 1u << 23; s += gridDim.x * blockDim.x) {
    const float b = make(s, e), y = rcp_round(b);
    for (unsigned k = 0; k < 8u; ++k) {
      const unsigned h = mix(s * 8u + k + seed);
      // the first dividends have edge significands
      const unsigned t = k == 0u ? 0u : k == 1u ? 1u : k == 2u ? 0x7fffffu : h & 0x7fffffu;
      const float a = make(t, (int)(mix(h) % 120u) - 60);
      const float d = h >> 31 ? -a : a;
      note(r, d, b, mh_div(d, b, y), d / b);
    }
  }
}
extern "C" int run(int what, int e, unsigned seed, Result *out) {
  Result *r;
  if (cudaMalloc(&r, sizeof(Result)) != cudaSuccess) return 1;
  cudaMemset(r, 0, sizeof(Result));
  if (what < 2) k_unary<<<608, 256>>>(r, what, e);
  else k_quotient<<<608, 256>>>(r, e, seed);
  const cudaError_t launched = cudaGetLastError();
  const cudaError_t done = cudaMemcpy(out, r, sizeof(Result), cudaMemcpyDeviceToHost);
  cudaFree(r);
  return launched != cudaSuccess || done != cudaSuccess;
}
'''


class Result(C.Structure):
    _fields_ = [("wrong", C.c_uint64), ("a", C.c_float), ("b", C.c_float)]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("round")
    (d / "r.cu").write_text(SRC)
    subprocess.check_call([B.nvcc(), "-shared", "-I", B.CSRC, str(d / "r.cu"), "-o", str(d / "r.so")] + B.ARCH + B.FLAGS)
    return C.CDLL(os.path.join(str(d), "r.so"))


def _run(lib, what, e, seed=0):
    r = Result()
    assert lib.run(what, e, seed, C.byref(r)) == 0
    assert r.wrong == 0, f"{r.wrong} differ, one at a = {r.a!r}, b = {r.b!r}"


@pytest.mark.parametrize("e", [-80, -79, -60, -41, -2, -1, 0, 1, 2, 29, 59, 78, 79])
def test_reciprocal(lib, e):
    _run(lib, 0, e)


@pytest.mark.parametrize("e", [-80, -79, -60, -59, -2, -1, 0, 1, 2, 29, 59, 78, 79])
def test_square_root(lib, e):
    _run(lib, 1, e)


@pytest.mark.parametrize("e", [0, 1, 2, 7, 19, 28, 29])
def test_quotient(lib, e):
    for seed in range(4):
        _run(lib, 2, e, seed * 977)
