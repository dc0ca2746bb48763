"""The two forms of the PSDF update, against the FP32 oracle, bit for bit.

In small images and with large voxels the update goes over all candidates at once;
else it drops those that it cannot change first, and reads records of the pixels.
Images on both sides of that line, with the depths, poses and blocks of
test_gpu_psdf_select.py, and frames of both forms: a batch always selects, a single
volume only above the line.
"""
import numpy as np
import pytest

from meshhashing_gb300 import Batch, Volume, config, scene
from oracle.oracle import Oracle
from tests.test_gpu_psdf_select import POSES, _depth

pytestmark = pytest.mark.gpu


# at 4 mm images of more than 2560 pixels select, at 8 mm of more than 20480, at 12 mm of more than 69120
@pytest.mark.parametrize("w,h,voxel", [(64, 40, 0.004), (61, 47, 0.004), (64, 48, 0.004), (90, 31, 0.004),
                                       (160, 128, 0.008), (161, 128, 0.008), (321, 219, 0.012), (640, 480, 0.016)])
@pytest.mark.parametrize("compat", [0, 1])
def test_updated_voxels(built, w, h, voxel, compat):
    rng = np.random.default_rng(w)
    wl = scene.full_spline(2, width=w, height=h)
    p = config.params_for(wl, voxel_size=voxel, truncation=3 * voxel, value_capacity=1 << 14, bucket_count=1 << 13,
                          max_vertex_count=1 << 12, max_triangle_count=1 << 12, compat_arithmetic=compat)
    own = np.asarray(wl.pose(0), np.float64)
    updated = left_out = 0
    for name, move in POSES.items():
        wTc = move(own).astype(np.float32)
        z = rng.uniform(-0.5, 3.0, 4000)
        c = np.stack([z * rng.uniform(-0.8, 0.8, 4000), z * rng.uniform(-0.8, 0.8, 4000), z, np.ones(4000)], 1)
        pos = np.unique(np.floor((c @ wTc.T.astype(np.float64))[:, :3] / (8 * voxel)).astype(np.int32), axis=0)
        depth = _depth(w, h, "steps" if name == "own" else "smooth", rng)
        v, o = Volume(p), Oracle(p, fp64=False)
        for s in (v, o):
            (s.load_blocks if s is v else s.set_blocks)(pos, *[np.zeros((len(pos), 512), np.float32)] * 4)
        v.set_frame(depth, wTc)
        o.frame_set(depth, wTc)
        v.collect_all_blocks()
        o.collect_all()
        v.predict_outlier_ratio()
        o.predict_inlier()
        v.update_blocks_bayesian()
        o.integrate_psdf()
        (gp, gf), (op, *of) = v.dump_blocks(), o.blocks()
        of = dict(zip(("sdf", "w", "a", "b"), of))
        gi, oi = np.lexsort(gp.T), np.lexsort(op.T)
        np.testing.assert_array_equal(gp[gi], op[oi])
        for k in ("sdf", "w", "a", "b"):
            np.testing.assert_array_equal(gf[k][gi].view(np.uint32), of[k][oi].view(np.uint32), err_msg=f"{name} {k}")
        updated += int((gf["w"] > 0).any(1).sum())
        left_out += int((gf["w"] == 0).all(1).sum())
    assert updated > 20 and left_out > 20


@pytest.mark.parametrize("w,h,voxel", [(64, 40, 0.004), (64, 48, 0.004), (96, 72, 0.016)])
@pytest.mark.parametrize("compat", [0, 1])
def test_frames(built, w, h, voxel, compat):
    wl = scene.full_spline(12, width=w, height=h)
    p = config.params_for(wl, voxel_size=voxel, truncation=3 * voxel, value_capacity=1 << 17, bucket_count=1 << 16,
                          max_vertex_count=1 << 18, max_triangle_count=1 << 18, compat_arithmetic=compat)
    v, u = Volume(p), Volume(p)
    batch = Batch([u], raycast=False)
    for k in range(12):
        v.integrate_frame(wl.frame(k), wl.pose(k))
        batch.step([wl.frame(k)], [wl.pose(k)])
    (pa, fa), (pb, fb) = v.dump_blocks(), u.dump_blocks()
    ia, ib = np.lexsort(pa.T), np.lexsort(pb.T)
    np.testing.assert_array_equal(pa[ia], pb[ib])
    for key in fa:
        np.testing.assert_array_equal(fa[key][ia].view(np.uint32), fb[key][ib].view(np.uint32))
    np.testing.assert_array_equal(v.neg_masks(pa), u.neg_masks(pa))
    batch.close()
