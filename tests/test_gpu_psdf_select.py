"""The blocks that the PSDF update leaves out, against the FP32 oracle, bit for bit.

The update drops candidates that lie beside the image or behind everything in
it before it projects their voxels.  Empty blocks all around the camera show
each voxel that is updated: its fields become a function of its pixel alone,
without an exponential.  Ragged images, holes, steps and outliers in depth,
blocks behind the camera, at it and larger than the image, and matrices that
are not rigid.
"""
import numpy as np
import pytest

from meshhashing_gb300 import Volume, config, scene
from meshhashing_gb300.pose import left_update
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

POSES = {
    "own": lambda T: T,
    "turned": lambda T: left_update(T, [0.3, -0.2, 0.1, 0.5, -0.7, 0.4]),
    "far": lambda T: left_update(T, [900.0, -700.0, 30.0, 0.0, 0.0, 0.3]),
    "scaled": lambda T: T @ np.diag([1.2, 0.8, 1.1, 1.0]),
    "sheared": lambda T: T @ np.array([[1, 0.3, 0, 0], [0, 1, -0.2, 0], [0.1, 0, 1, 0], [0, 0, 0, 1.0]]),
}


def _depth(w, h, kind, rng):
    y, x = np.mgrid[0:h, 0:w]
    d = 1.0 + 0.6 * np.sin(x / 9.0) + 0.4 * np.cos(y / 7.0)
    if kind == "steps":
        d = np.where((x // 6 + y // 5) % 2 == 0, 0.7, 2.6)
    d = d + rng.normal(0.0, 0.003, d.shape)
    holes, out = rng.random(d.shape) < 0.1, rng.random(d.shape) < 0.01
    return np.where(holes, 0.0, np.where(out, rng.uniform(0.3, 5.0, d.shape), d)).astype(np.float32)


@pytest.mark.parametrize("w,h,voxel", [(1, 1, 0.02), (7, 5, 0.02), (64, 48, 0.008), (61, 47, 0.03), (64, 48, 0.2)])
def test_updated_voxels(built, w, h, voxel):
    rng = np.random.default_rng(w)
    wl = scene.full_spline(2, width=w, height=h)
    p = config.params_for(wl, voxel_size=voxel, truncation=3 * voxel, value_capacity=1 << 14, bucket_count=1 << 13,
                          max_vertex_count=1 << 12, max_triangle_count=1 << 12)
    own = np.asarray(wl.pose(0), np.float64)
    updated = left_out = 0
    for name, move in POSES.items():
        wTc = move(own).astype(np.float32)
        # blocks along the rays to 3 m and around the camera
        z = rng.uniform(-0.5, 3.0, 4000)
        c = np.stack([z * rng.uniform(-0.8, 0.8, 4000), z * rng.uniform(-0.8, 0.8, 4000), z, np.ones(4000)], 1)
        pos = np.unique(np.floor((c @ wTc.T.astype(np.float64))[:, :3] / (8 * voxel)).astype(np.int32), axis=0)
        for kind in ("smooth", "steps"):
            depth = _depth(w, h, kind, rng)
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
