"""The raycast's grid of cells and blocks against the FP32 oracle, bit for bit.

The grid follows the view: cells of 2 voxels, or larger where the image is
small (128 words a pixel), blocks from a dense array, or from the hash table
where the view holds too many.  Images with ragged tiles, poses on and off the
map, outside it and looking away, matrices that are not rigid, and more
raycasts than the dense array has tags.
"""
import numpy as np
import pytest

from meshhashing_gb300 import Volume, config, scene
from meshhashing_gb300.pose import left_update
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

POSES = {
    "own": lambda T: T,
    "moved": lambda T: left_update(T, [0.1, -0.07, 0.05, 0.1, 0.2, -0.15]),
    "outside": lambda T: left_update(T, [3.0, -2.0, 0.4, 0.0, 0.0, 2.5]),
    "away": lambda T: left_update(T, [40.0, 40.0, 0.0, 0.0, 0.0, 0.0]),
    "scaled": lambda T: T @ np.diag([1.2, 0.8, 1.1, 1.0]),
}


def _map(w, h, voxel, frames=6, **over):
    wl = scene.full_spline(frames, width=w, height=h)
    p = config.params_for(wl, voxel_size=voxel, truncation=3 * voxel, value_capacity=1 << 16, bucket_count=1 << 16,
                          max_vertex_count=1 << 16, max_triangle_count=1 << 16, **over)
    v = Volume(p)
    for i in range(frames):
        v.integrate_frame(wl.frame(i), wl.pose(i))
    o = Oracle(p, fp64=False)
    pos, f = v.dump_blocks()
    o.set_blocks(pos, f["sdf"], f["w"], f["a"], f["b"])
    assert v.stats()["error"] == 0
    return wl, v, o


def _same(v, o, cTw):
    gd, gv, gn = v.raycast(cTw)
    od, ov, on = o.raycast(cTw)
    for g, r in ((gd, od), (gv, ov), (gn, on)):
        hit = np.isfinite(r)
        assert np.array_equal(np.isfinite(g), hit)
        np.testing.assert_array_equal(g[hit].view(np.uint32), r[hit].view(np.uint32))
    return int(np.isfinite(od).sum())


# cells of 8, 4, 2 and 8 voxels; at 1 mm 32, and the blocks come from the hash table
@pytest.mark.parametrize("w,h,voxel", [(36, 28, 0.004), (124, 92, 0.004), (124, 92, 0.008), (52, 44, 0.0047),
                                       (40, 28, 0.001)])
def test_views(built, w, h, voxel):
    wl, v, o = _map(w, h, voxel)
    hits = {}
    for name, move in POSES.items():
        T = move(np.asarray(wl.pose(5), np.float64))
        hits[name] = _same(v, o, np.linalg.inv(T).astype(np.float32))
    assert hits["own"] > w * h // 4 and hits["away"] == 0
    assert v.stats()["error"] == 0


def test_more_raycasts_than_tags(built):
    wl, v, o = _map(36, 28, 0.008)
    poses = [np.linalg.inv(left_update(np.asarray(wl.pose(5), np.float64), [0.3 * s, 0.0, 0.0, 0.0, 0.0, 0.4 * s]))
             .astype(np.float32) for s in (-1.0, 0.0, 1.0)]
    first = [v.raycast(c) for c in poses]
    for k in range(90):
        for c, ref in zip(poses, first):
            for a, b in zip(v.raycast(c), ref):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), k
    assert _same(v, o, poses[1]) > 0


@pytest.mark.parametrize("w,h", [(37, 29), (33, 30), (31, 29)])
def test_host_images_of_any_size(built, w, h):
    """Pixel counts of 1, 2 and 3 modulo 4: the staged vertices and normals are vectors of four."""
    assert (w * h) % 4 == {37: 1, 33: 2, 31: 3}[w]
    wl, v, o = _map(w, h, 0.008)
    T = np.asarray(wl.pose(5), np.float64)
    assert _same(v, o, np.linalg.inv(T).astype(np.float32)) > 0


# The last and first images of 8, 4 and 1 lanes a ray, whole and ragged tiles.
@pytest.mark.parametrize("w,h", [(1, 1), (5, 3), (256, 256), (257, 256), (512, 256), (513, 256)])
def test_lanes_of_a_ray(built, w, h):
    wl, v, o = _map(w, h, 0.016)
    T = np.asarray(wl.pose(5), np.float64)
    hits = [_same(v, o, np.linalg.inv(m(T)).astype(np.float32)) for m in (POSES["own"], POSES["moved"])]
    assert hits[0] > w * h // 4 or w * h < 100


# Steps that lie halfway between two floats: t + step rounds down and up in turn
# from 0.25 m, 0.5 m or 1 m on, so its samples have no closed form there.
@pytest.mark.parametrize("half", [2.0 ** -26, 2.0 ** -25, 2.0 ** -24])
def test_steps_that_round_both_ways(built, half):
    wl, v, o = _map(60, 44, 0.008, raycast_step=2.0 ** -7 + half)
    T = np.asarray(wl.pose(5), np.float64)
    assert _same(v, o, np.linalg.inv(T).astype(np.float32)) > 60 * 44 // 4


# One grid serves a refinement's poses where it covers them: the last pass's sums
# against those of a grid made for that pose alone.  Its inverse may differ by
# units in the last place, 1e-6 m of depth, which moves a pixel in a thousand
# across the gate at most.
@pytest.mark.parametrize("w,h,voxel", [(64, 48, 0.008), (124, 92, 0.004), (40, 28, 0.001)])
@pytest.mark.parametrize("off", [0.0, 0.01, 0.3])
def test_refinement_on_one_grid(built, w, h, voxel, off):
    wl, v, o = _map(w, h, voxel)
    T = np.asarray(wl.pose(5), np.float64)
    v.set_frame(wl.frame(5), T)
    start = left_update(T, [off, -off, 0.5 * off, -off, 0.7 * off, off])
    for n in (0, 1, 6):
        T1, cost, count = v.refine_pose(start, iterations=n, max_residual=0.05)
        _, _, cost2, count2 = v.normal_equations(np.linalg.inv(T1.astype(np.float64)).astype(np.float32),
                                                 max_residual=0.05)
        assert abs(count - count2) <= 2 + 1e-3 * w * h
        assert abs(cost - cost2) <= 1e-3 * cost2 + 3 * 0.05 ** 2
        assert off > 0.1 or count > 0
