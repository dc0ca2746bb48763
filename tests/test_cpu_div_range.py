"""Quotients by a known divisor over the whole range that csrc/mh_div.h states.

Divisors of 2^-60 .. 2^60, far beyond any voxel size, with dividends up to the
limits of mh_div_ok: nothing over- or underflows there, so every quotient is the
rounded one.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = '''
#include "mh_div.h"
extern "C" void quotients(const float *a, int n, float b, float *mine, float *exact) {
  const float y = 1.0f / b;
  for (int i = 0; i < n; ++i) mine[i] = mh_div(a[i], b, y), exact[i] = a[i] / b;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("divrange")
    (d / "q.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "meshhashing_gb300", "csrc"), str(d / "q.cpp"), "-o", str(d / "q.so")])
    return C.CDLL(str(d / "q.so"))


@pytest.mark.parametrize("e", [-60, -59, -45, -30, -21, 20, 21, 30, 45, 58, 59])
def test_quotients_are_rounded(lib, e):
    rng = np.random.default_rng(e + 100)
    edge = np.array([1.0, 1.0 + 2.0 ** -23, 2.0 - 2.0 ** -23, 1.5, 1.5 - 2.0 ** -23, 1.5 + 2.0 ** -23])
    for s in np.concatenate([edge, 1.0 + rng.integers(0, 1 << 23, 10) * 2.0 ** -23]):
        b = np.float32(np.ldexp(s, e))
        sig = np.concatenate([edge, 1.0 + rng.integers(0, 1 << 23, 20000) * 2.0 ** -23]).astype(np.float32)
        exp = rng.choice([-60, -59, -40, -1, 0, 1, 40, 58, 59], sig.size)
        a = np.ldexp(sig, exp).astype(np.float32)
        a = a[(a > 1e-18) & (a < 1e18)]
        mine, exact = np.empty_like(a), np.empty_like(a)
        p = lambda x: x.ctypes.data_as(C.c_void_p)  # noqa: E731
        lib.quotients(p(a), a.size, C.c_float(b), p(mine), p(exact))
        np.testing.assert_array_equal(mine.view(np.uint32), exact.view(np.uint32))
