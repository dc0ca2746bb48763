"""The view grid's host side (csrc/mh_ray_grid.h), compiled for the host.

A grid asks for the block array's clear when the memory is new or its tags have
started over.  A caller may drop a grid before anything of it is enqueued; the
clear has to stay due until it is.  Where a buffer cannot be allocated there is a
grid without it, or none.
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from meshhashing_gb300 import config, scene

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = '''
#include "mh_ray_grid.h"
static mh_params P;
static RayGridBuf B;
static unsigned memory[1];
extern "C" void set_up(const mh_params *p) {
  P = *p;
  B = RayGridBuf{};
  ray_grid_sizes(P, B);
  B.bits = B.blocks = memory;  // not written here
}
extern "C" unsigned entries() { return B.entries; }
// the grid of a volume of which the first `have` buffers could be allocated, the number of buffers asked for
extern "C" int reserve(const mh_params *p, const float *wTc, int have, int *cells, int *blocks) {
  RayGridBuf b;
  int asked = 0;
  for (int k = 0; k < 2; ++k)
    ray_grid_reserve(*p, b, [&](unsigned words) { return words && asked++ < have ? memory : (unsigned *)nullptr; });
  const RayGrid g = ray_grid_for(*p, wTc, b);
  *cells = g.bits != nullptr;
  *blocks = g.blocks != nullptr;
  return asked;
}
extern "C" void draw(const float *wTc, int enqueue, unsigned *tag, unsigned *clear) {
  const RayGrid g = ray_grid_for(P, wTc, B);
  *tag = g.tag >> 24;
  *clear = g.clear;
  if (enqueue) ray_grid_enqueued(B, g);
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("grid")
    (d / "g.cpp").write_text(SRC)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                           os.path.join(ROOT, "meshhashing_gb300", "csrc"), str(d / "g.cpp"), "-o", str(d / "g.so")])
    return C.CDLL(str(d / "g.so"))


def _draws(lib, enqueued):
    wl = scene.full_spline(2, width=36, height=28)
    p = config.params_for(wl, voxel_size=0.008, truncation=0.024, value_capacity=1 << 16)
    lib.set_up(C.byref(p))
    T = np.ascontiguousarray(np.asarray(wl.pose(1), np.float32).reshape(16))
    out = []
    for ok in enqueued:
        tag, clear = C.c_uint(), C.c_uint()
        lib.draw(T.ctypes.data_as(C.c_void_p), int(ok), C.byref(tag), C.byref(clear))
        out.append((tag.value, clear.value))
    assert lib.entries() > 0
    return out, lib.entries()


def _stale_read(lib, enqueued):
    """Whether a raycast that was enqueued finds entries with its tag that an
    earlier raycast, or the memory's last owner, left."""
    draws, entries = _draws(lib, enqueued)
    left = set(range(256))               # tags that the array may hold
    for (tag, clear), ok in zip(draws, enqueued):
        assert 1 <= tag < 255 and clear in (0, entries)
        if not ok:
            continue
        if clear:
            left = set()
        if tag in left:
            return True
        left.add(tag)
    return False


@pytest.mark.parametrize("lost", [[], [0], [0, 1], [253], [254], [255], [252, 253, 254, 255, 256],
                                  [0, 253, 254, 507, 508, 509, 510], list(range(0, 800, 3))])
def test_clear_stays_due(lib, lost):
    assert not _stale_read(lib, [k not in lost for k in range(800)])


def test_a_clear_is_asked_for_once(lib):
    draws, entries = _draws(lib, [True] * 600)
    clears = [k for k, (_, clear) in enumerate(draws) if clear]
    assert clears[0] == 0 and len(clears) == 3 and all(b - a >= 250 for a, b in zip(clears, clears[1:]))


@pytest.mark.parametrize("have,cells,blocks,asked", [(0, 0, 0, 1), (1, 1, 0, 2), (2, 1, 1, 2)])
def test_a_grid_without_memory(lib, have, cells, blocks, asked):
    wl = scene.full_spline(2, width=36, height=28)
    p = config.params_for(wl, voxel_size=0.008, truncation=0.024, value_capacity=1 << 16)
    T = np.ascontiguousarray(np.asarray(wl.pose(1), np.float32).reshape(16))
    c, b = C.c_int(), C.c_int()
    n = lib.reserve(C.byref(p), T.ctypes.data_as(C.c_void_p), have, C.byref(c), C.byref(b))
    assert (c.value, b.value, n) == (cells, blocks, asked)
