"""Voxels that are unobserved for some Huber-TV calls keep their state.

An init, then calls between which some voxels lose their weight and get it back:
their extrapolated sdf and dual are those of the last call that updated them.
Against the FP32 oracle; the data weight is exp() of two libraries, a few units in
the last place apart (2e-6 of the field's range).
"""
import numpy as np
import pytest

from meshhashing_gb300 import Volume, config, scene
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.02, 0.3, 1.0])
@pytest.mark.parametrize("cells", [[(0, 0, 0)], [(x, y, z) for x in range(2) for y in range(2) for z in range(2)]])
def test_weights_that_come_back(built, cells, share):
    wl = scene.small_circle(4)
    p = config.params_for(wl, value_capacity=1 << 10, bucket_count=1 << 10, max_vertex_count=1 << 10,
                          max_triangle_count=1 << 10)
    rng = np.random.default_rng(7)
    pos = np.array(cells, np.int32)
    sdf = rng.uniform(-0.02, 0.02, (len(cells), 512)).astype(np.float32)
    w = np.full_like(sdf, 5.0)
    away = np.where(rng.random(w.shape) < share, 0.0, w).astype(np.float32)
    v, o = Volume(p), Oracle(p, fp64=False)
    v.load_blocks(pos, sdf, w)
    o.set_blocks(pos, sdf, w, np.zeros_like(w), np.zeros_like(w))
    for x in (v, o):
        x.set_candidates(pos)
        x.huber_tv_init()
    for weights in (w, away, w, away, w):
        v.load_blocks(pos, None, weights)
        o.set_blocks(pos, None, weights)
        e, eo = v.huber_tv_iterate(2.0, 8.0, 0.01, 2), o.huber_tv_iterate(2.0, 8.0, 0.01, 2)
        np.testing.assert_allclose(e, eo, rtol=1e-4, atol=1e-30)
        gp, gf = v.dump_blocks(("sdf",))
        op, of = o.blocks()[:2]
        got, want = gf["sdf"][np.lexsort(gp.T)], of[np.lexsort(op.T)]
        np.testing.assert_allclose(got, want, rtol=0, atol=2e-6 * np.abs(sdf).max())
