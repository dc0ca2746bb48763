"""Views whose grid has large cells, and views far from the origin, against the
FP32 oracle, bit for bit.

A small image at fine voxels gets cells of up to 128 voxels; kilometres from the
origin the positions' roundings come near a voxel.  Both move samples across the
cells' borders.  The maps are volumes of positive voxels, with a negative plate just
above such a border (the plane through the world's origin is one for every cell
size) or with negative blobs everywhere, and the march takes half-voxel steps: one
sample skipped too many changes a hit.
"""
import numpy as np
import pytest

from meshhashing_gb300 import Volume, config, scene
from meshhashing_gb300.pose import left_update
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _map(w, h, voxel, origin, step):
    wl = scene.full_spline(2, width=w, height=h)
    p = config.params_for(wl, voxel_size=voxel, truncation=3 * voxel, value_capacity=1 << 14, bucket_count=1 << 14,
                          max_vertex_count=1 << 12, max_triangle_count=1 << 12, raycast_step=step)
    n = 24
    pos = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    rng = np.random.default_rng(5)
    s = 8 * n
    field = rng.uniform(0.2, 1.0, (s, s, s)).astype(np.float32) * np.float32(2 * voxel)   # z, y, x
    for c in rng.integers(0, s - 2, (4000, 3)):
        field[c[0]:c[0] + 2, c[1]:c[1] + 2, c[2]:c[2] + 2] *= np.float32(-1.0)
    sdf = np.stack([field[8 * z:8 * z + 8, 8 * y:8 * y + 8, 8 * x:8 * x + 8].reshape(512) for x, y, z in pos])
    side = 8.0 * voxel
    first = np.floor((np.asarray(origin) + np.array([-0.5 * n * side, -0.5 * n * side, 0.6])) / side).astype(np.int64)
    pos = (pos + first).astype(np.int32)
    w = np.ones_like(sdf)
    v, o = Volume(p), Oracle(p, fp64=False)
    v.load_blocks(pos, sdf, w)
    o.set_blocks(pos, sdf, w, np.zeros_like(w), np.zeros_like(w))
    return v, o


def _poses(origin, count):
    rng = np.random.default_rng(11)
    for _ in range(count):
        T = left_update(np.eye(4), np.concatenate([rng.uniform(-0.05, 0.05, 3), rng.uniform(-0.2, 0.2, 3)]))
        T[:3, 3] += origin
        yield np.linalg.inv(T).astype(np.float32)


def _same(v, o, cTw):
    hits = 0
    for g, r in zip(v.raycast(cTw), o.raycast(cTw)):
        hit = np.isfinite(r)
        assert np.array_equal(np.isfinite(g), hit)
        np.testing.assert_array_equal(g[hit].view(np.uint32), r[hit].view(np.uint32))
        hits += int(hit.sum())
    return hits


# cells of 32, 64, 64, 128 and 128 voxels; the plate's first layer from the border
@pytest.mark.parametrize("w,h,voxel,layers", [(16, 12, 0.004, 4), (16, 12, 0.002, 6), (40, 28, 0.001, 6),
                                              (16, 12, 0.001, 9), (5, 3, 0.001, 9)])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_plate_above_a_border(built, w, h, voxel, layers, axis):
    wl = scene.full_spline(2, width=w, height=h)
    p = config.params_for(wl, voxel_size=voxel, truncation=3 * voxel, value_capacity=1 << 14, bucket_count=1 << 14,
                          max_vertex_count=1 << 12, max_triangle_count=1 << 12, raycast_step=0.5 * voxel)
    half = np.full(3, 10)
    half[axis] = 4
    pos = np.stack(np.meshgrid(*[np.arange(-k, k) for k in half], indexing="ij"), -1).reshape(-1, 3).astype(np.int32)
    at = 8 * pos[:, None, axis] + (np.arange(512) >> 3 * axis & 7)     # voxel coordinate across the plate
    v, o = Volume(p), Oracle(p, fp64=False)
    ones = np.ones((len(pos), 512), np.float32)
    rng = np.random.default_rng(axis)
    hits = 0
    for first in range(layers):
        sdf = np.where((at == first) | (at == first + 1), -3.0 * voxel, 1.0 * voxel).astype(np.float32)
        v.load_blocks(pos, sdf, ones)
        o.set_blocks(pos, sdf, ones, 0 * ones, 0 * ones)
        for sign in (1.0, -1.0):
            for _ in range(10):
                z = np.zeros(3)
                z[axis] = sign
                x = np.roll(z, 1)
                T = np.eye(4)
                T[:3, :3] = np.stack([x, np.cross(z, x), z], 1)
                T[:3, 3] = -z * (32.0 * voxel + 0.52 + 0.05 * rng.random())
                T = T @ left_update(np.eye(4), np.concatenate([rng.uniform(-0.01, 0.01, 3), rng.uniform(-0.1, 0.1, 3)]))
                hits += _same(v, o, np.linalg.inv(T).astype(np.float32))
    assert hits > 0 and v.stats()["error"] == 0


# offsets on all axes, in metres; the images' cells are of 2 voxels and up
@pytest.mark.parametrize("off", [60.0, 900.0, 3000.0, 5000.0, 20000.0, 50000.0])
@pytest.mark.parametrize("w,h,voxel", [(124, 92, 0.008), (36, 28, 0.008)])
def test_far_from_the_origin(built, w, h, voxel, off):
    origin = np.array([off, -0.7 * off, 0.9 * off])
    v, o = _map(w, h, voxel, origin, 0.5 * voxel)
    hits = sum(_same(v, o, c) for c in _poses(origin, 4))
    assert hits > 0 or off > 10000.0
    assert v.stats()["error"] == 0
