"""Marching cubes and the low-surfel flags on random blocks against the FP32 oracle.

Random signs put vertices on most edges, so owners on every face, edge and
corner of a block are marked by one, two or four blocks, and gaps between the
blocks leave samples without a neighbour.  A second and third pass with other
values reuse, free and allocate vertices, triangles and pages.
"""
import numpy as np
import pytest

from meshhashing_gb300 import Volume, config, scene
from oracle.oracle import Oracle
from tests._util import mesh_canon

pytestmark = pytest.mark.gpu


def _blocks(side, keep, rng):
    g = np.stack(np.meshgrid(*[np.arange(-side // 2, side - side // 2)] * 3, indexing="ij"), -1).reshape(-1, 3)
    return g[rng.random(len(g)) < keep].astype(np.int32)


def _values(n, voxel, flat, rng):
    shape = (n, 512)
    sdf = rng.uniform(-2 * voxel, 2 * voxel, shape)
    # `flat` of the blocks have no sign change: no page, or theirs is given back
    sdf[rng.random(n) < flat] = voxel
    w = rng.uniform(0.97, 3.0, shape) / voxel ** 2
    a = rng.uniform(0.5, 9.0, shape)
    return [x.astype(np.float32) for x in (sdf, w, a, np.ones(shape))]


@pytest.mark.parametrize("side,keep,flat,voxel", [(1, 1.0, 0.0, 0.008), (4, 1.0, 0.5, 0.008), (7, 0.6, 0.3, 0.0047),
                                                  (14, 0.35, 0.6, 0.02)])
def test_random_blocks(built, side, keep, flat, voxel):
    rng = np.random.default_rng(side)
    wl = scene.full_spline(1, width=64, height=48)
    p = config.params_for(wl, voxel_size=voxel, truncation=3 * voxel, value_capacity=1 << 13, bucket_count=1 << 12,
                          max_vertex_count=1 << 20, max_triangle_count=1 << 21)
    v, o = Volume(p), Oracle(p, fp64=False)
    pos = _blocks(side, keep, rng)
    count = 0
    for k in range(3):
        f = _values(len(pos), voxel, flat, rng)
        v.load_blocks(pos, *f)
        o.set_blocks(pos, *f)
        # in the second pass a part of the blocks, so the others get pages but no pass
        cand = pos if k != 1 else pos[rng.random(len(pos)) < 0.7]
        v.set_candidates(cand)
        o.set_candidates(cand)
        v.marching_cubes()
        o.mesh()
        gv, gt = mesh_canon(*v.dump_mesh())
        ov, ot = mesh_canon(*o.dump_mesh())
        assert set(gv) == set(ov) and gt == ot
        for m in range(3):
            np.testing.assert_array_equal(v.block_meta(cand)[m], o.block_meta(cand)[m])
        if gv:
            # the same operations in the same order and precision
            a, b = np.stack([gv[q] for q in sorted(gv)]), np.stack([ov[q] for q in sorted(ov)])
            np.testing.assert_array_equal(a, b)
        count += len(gt)
        v.collect_low_surfel_blocks()
        o.gc_low_surfel()
        flags = {tuple(c): int(x) for c, x in zip(v.candidates(), v.flags())}
        assert flags == {tuple(c): int(x) for c, x in zip(cand, o.block_meta(cand)[3])}
    assert count > 0 and v.stats()["error"] == 0
