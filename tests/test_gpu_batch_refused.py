"""A batch step that is refused changes nothing.

The second scene's depth is missing, so the step is refused after the first
scene's turn.  The first scene's raycasts that follow must not take old entries
of its view's block array as blocks: not in memory that another volume has used,
and not where the array's tags start over (254 raycasts).  Every later step
equals the single volumes' bit for bit, frame counters included.
"""
import gc

import numpy as np
import pytest

from meshhashing_gb300 import Batch, Volume, config, scene
from meshhashing_gb300._lib import MeshHashError

pytestmark = pytest.mark.gpu


def _spec(seed):
    wl = scene.full_spline(24, width=48, height=36, seed=seed)
    return wl, config.params_for(wl, voxel_size=0.016, truncation=0.048, value_capacity=1 << 13, bucket_count=1 << 12,
                                 max_vertex_count=1 << 16, max_triangle_count=1 << 16)


def _cTw(wl, k):
    return np.linalg.inv(np.asarray(wl.pose(k), np.float64)).astype(np.float32)


@pytest.mark.parametrize("before", [0, 252, 253, 254, 255])
@pytest.mark.parametrize("graph", [False, True])
def test_refused_step(built, before, graph):
    specs = [_spec(0), _spec(3)]
    # the memory's last owner: its block array holds entries of many tags
    wl, p = specs[0]
    last = Volume(p)
    for k in range(4):
        last.integrate_frame(wl.frame(k), wl.pose(k))
    for k in range(260):
        last.raycast(_cTw(wl, k % 4))
    last.close()
    del last
    gc.collect()
    batched = [Volume(p) for _, p in specs]
    singles = [Volume(p) for _, p in specs]
    for v, (wl, _) in zip(batched, specs):
        for k in range(before):
            v.raycast(_cTw(wl, k % 8))
    batch = Batch(batched, raycast=True)
    for k in range(12):
        if k in (0, 1, 5):
            with pytest.raises(MeshHashError):
                batch.step([specs[0][0].frame(k), None], [wl.pose(k) for wl, _ in specs], use_graph=graph)
            assert [v.stats()["frames"] for v in batched] == [k, k]
        batch.step([wl.frame(k) for wl, _ in specs], [wl.pose(k) for wl, _ in specs], use_graph=graph)
        for i, (wl, p) in enumerate(specs):
            d = np.empty((p.rc_height, p.rc_width), np.float32)
            n = np.empty((p.rc_height, p.rc_width, 4), np.float32)
            singles[i].integrate_frame(wl.frame(k), wl.pose(k), ray_depth=d, ray_normal=n)
            bd, _, bn = batch.raycast(i)
            np.testing.assert_array_equal(bd.view(np.uint32), d.view(np.uint32))
            np.testing.assert_array_equal(bn.view(np.uint32), n.view(np.uint32))
    for a, b in zip(batched, singles):
        (pa, fa), (pb, fb) = a.dump_blocks(), b.dump_blocks()
        ia, ib = np.lexsort(pa.T), np.lexsort(pb.T)
        np.testing.assert_array_equal(pa[ia], pb[ib])
        for key in fa:
            np.testing.assert_array_equal(fa[key][ia].view(np.uint32), fb[key][ib].view(np.uint32))
        sa, sb = a.stats(), b.stats()
        assert sa["frames"] == sb["frames"] == 12 and sa["error"] == sb["error"] == 0
        assert sa["gc_freed_blocks"] == sb["gc_freed_blocks"]
    batch.close()
