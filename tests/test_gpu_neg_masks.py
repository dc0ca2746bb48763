"""The blocks' masks of voxels that may not be non-negative, after each writer.

The raycast steps over cells, and the mesh pass leaves out blocks, that no set bit
touches (mh_dump_neg_masks), so no clear bit may lie over a voxel whose sdf is
outside [0, 1e30).  Checked against the voxels themselves after the simple and the
PSDF update, the collections that free blocks and hand them out again, Huber-TV,
loaded blocks and checkpoints, a reset and a batch.
"""
import numpy as np
import pytest

from meshhashing_gb300 import Batch, Volume, config, scene
from tests._neg_masks import hidden, needed

pytestmark = pytest.mark.gpu


def _check(v, what):
    pos, f = v.dump_blocks(("sdf",))
    mask = v.neg_masks(pos)
    bad = hidden(f["sdf"], mask)
    assert bad.size == 0, f"{what}: masks of {bad.size} of {len(pos)} blocks hide a voxel"
    return int((needed(f["sdf"]) != 0).sum()), int((mask != 0).sum()), len(pos)


def _psdf(frames=24, **over):
    wl = scene.full_spline(frames, width=160, height=120)
    return wl, config.params_for(wl, voxel_size=0.006, truncation=0.018, value_capacity=1 << 17, bucket_count=1 << 16,
                                 max_vertex_count=1 << 19, max_triangle_count=1 << 19, **over)


@pytest.mark.parametrize("compat", [0, 1])
def test_psdf_chain_and_huber(built, compat):
    wl, p = _psdf()
    p.compat_arithmetic = compat
    v = Volume(p)
    for k in range(21):                        # blocks are freed at frames 10 and 20
        v.integrate_frame(wl.frame(k), wl.pose(k), tv_iterations=5 if k % 2 else 0)
        if k in (0, 9, 10, 20):
            _check(v, f"frame {k}")
    assert v.stats()["gc_freed_blocks"] > 0
    need, have, total = _check(v, "PSDF chain")
    assert 0 < need <= have < total
    v.huber_tv_init()
    for _ in range(3):
        v.huber_tv_iterate(2.0, 8.0, 0.05, 4)
        _check(v, "Huber-TV")
    v.collect_all_blocks()                     # blocks of all kinds, unobserved voxels
    v.huber_tv_init()
    v.huber_tv_iterate(2.0, 8.0, 0.05, 4)
    _check(v, "Huber-TV over all blocks")


def test_simple_chain_with_starvation(built):
    wl = scene.small_circle(48)
    f = 262.5 * 160 / 320
    wl.camera = scene.Camera(160, 120, f, f, 79.5, 59.5)
    v = Volume(config.params_for(wl, value_capacity=1 << 16, bucket_count=1 << 15))
    for k in range(45):                        # starvation at frames 14, 29 and 44
        v.integrate_frame(wl.frame(k), wl.pose(k))
        if k % 5 == 4:
            _check(v, f"frame {k}")
    need, have, total = _check(v, "simple chain")
    assert 0 < need <= have < total


def test_freed_blocks_start_clear(built):
    """A pool that is nearly full hands out blocks again that held negative voxels."""
    wl, p = _psdf()
    v = Volume(p)
    for k in range(3):
        v.integrate_frame(wl.frame(k), wl.pose(k))
    used = v.stats()["block_high_water"]
    for _ in range(6):
        v.collect_all_blocks()
        v.starve_occupied_block_array()
        v.collect_low_surfel_blocks()
        v.collect_garbage_block_array()
        v.recycle_garbage_block_array()
        _check(v, "collection")
    assert v.stats()["gc_freed_blocks"] > 0
    for k in range(12, 15):
        v.integrate_frame(wl.frame(k), wl.pose(k))
        _check(v, "after a collection")
    assert v.stats()["block_high_water"] <= 2 * used and v.stats()["error"] == 0


def test_loaded_blocks_checkpoint_and_reset(built, tmp_path):
    wl, p = _psdf(4)
    v = Volume(p)
    # a voxel at every place, of every kind, with all others non-negative
    pos = np.array([(i, 3 * i % 7, -i) for i in range(512)], np.int32)
    rng = np.random.default_rng(1)
    sdf = rng.uniform(0.0, 0.02, (512, 512)).astype(np.float32)
    for i, value in enumerate(np.tile(np.array([-1e-30, -0.01, np.nan, np.inf, -np.inf, 1e30], np.float32), 86)[:512]):
        sdf[i, i] = value
    w = np.ones_like(sdf)
    v.load_blocks(pos, sdf, w)
    np.testing.assert_array_equal(v.neg_masks(pos), needed(sdf))
    v.load_blocks(pos, np.abs(np.nan_to_num(sdf, posinf=0.0, neginf=0.0)) % np.float32(1.0))   # the same blocks again
    assert not v.neg_masks(pos).any()
    v.load_blocks(pos, None, w)                # no sdf: the masks stay
    v.load_blocks(pos[::2], -sdf[::2])
    np.testing.assert_array_equal(v.neg_masks(pos[::2]), needed(-sdf[::2]))
    assert not v.neg_masks(pos[1::2]).any()
    path = str(tmp_path / "map.mhv")
    v.save(path)
    u = Volume(p)
    assert u.load(path) == len(pos)
    np.testing.assert_array_equal(u.neg_masks(pos), v.neg_masks(pos))
    _check(u, "checkpoint")
    v.reset()
    assert (v.neg_masks(pos) == np.uint64(2 ** 64 - 1)).all()   # no such block
    v.load_blocks(pos, None, w)                # new blocks hold sdf 0
    assert not v.neg_masks(pos).any()


def test_batch(built):
    specs = [_psdf(16), _psdf(16, bayesian=False)]
    vols = [Volume(p) for _, p in specs]
    batch = Batch(vols, raycast=False)
    for k in range(15):
        batch.step([wl.frame(k) for wl, _ in specs], [wl.pose(k) for wl, _ in specs], use_graph=k > 2)
    for v in vols:
        need, have, total = _check(v, "batch")
        assert 0 < need <= have <= total
    batch.close()
