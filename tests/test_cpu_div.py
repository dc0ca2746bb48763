"""Quotients by a known divisor (csrc/mh_div.h) are the rounded quotients.

Random and boundary significands (1, 1 + ulp, 2 - ulp, 1.5) of dividend and
divisor over the exponents that voxel coordinates take, against the compiler's
division; the header is compiled for the host with fused multiply-adds from
the C library.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = '''
#include "mh_div.h"
extern "C" void quotients(const float *a, int n, float b, float *mine, float *exact, int *ok) {
  const float y = 1.0f / b;
  for (int i = 0; i < n; ++i) {
    mine[i] = mh_div(a[i], b, y);
    exact[i] = a[i] / b;
    ok[i] = mh_div_ok(a[i], 1.0f, a[i]);
  }
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "q.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "meshhashing_gb300", "csrc"), str(d / "q.cpp"), "-o", str(d / "q.so")])
    return ctypes.CDLL(str(d / "q.so"))


def significands(rng, n):
    edge = np.array([1.0, 1.0 + 2.0 ** -23, 2.0 - 2.0 ** -23, 1.5, 1.5 - 2.0 ** -23, 1.5 + 2.0 ** -23])
    return np.concatenate([edge, 1.0 + rng.integers(0, 1 << 23, n) * 2.0 ** -23]).astype(np.float32)


@pytest.mark.parametrize("b", [0.004, 0.005, 0.006, 0.008, 0.001, 0.0047, 1.0, 2.0 ** -20, 2.0 ** 20 - 1.0])
def test_quotients_are_rounded(lib, b):
    rng = np.random.default_rng(int(b * 1e6) & 0xffff)
    for db in significands(rng, 8):
        div = np.float32(b) if db == 1.0 else np.float32(db * 2.0 ** np.floor(np.log2(b)))
        a = np.ldexp(significands(rng, 20000), rng.integers(-59, 59, 20006)).astype(np.float32)
        a *= rng.choice(np.array([-1.0, 1.0], np.float32), a.size)
        mine, exact, ok = np.empty_like(a), np.empty_like(a), np.empty(a.size, np.int32)
        p = lambda x: x.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
        lib.quotients(p(a), a.size, ctypes.c_float(div), p(mine), p(exact), p(ok))
        inside = (np.abs(a) > 1e-18) & (np.abs(a) < 1e18)
        np.testing.assert_array_equal(ok != 0, inside)
        np.testing.assert_array_equal(mine[inside].view(np.uint32), exact[inside].view(np.uint32))
