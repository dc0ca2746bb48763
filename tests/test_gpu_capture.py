"""Calls that a caller's CUDA graph replays give what the calls themselves give.

The launches are recorded once; the pose, the map and the work lists are those of
each replay.  Bit for bit against the same calls made without a graph, after the
pose has changed, after blocks have been freed between two replays, and with other
raycasts of the volume in between.
"""
import numpy as np
import pytest

from meshhashing_gb300 import Volume, config, scene
from meshhashing_gb300.pose import left_update

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _cTw(T):
    return np.linalg.inv(np.asarray(T, np.float64)).astype(np.float32)


def _params(wl, voxel, **over):
    return config.params_for(wl, voxel_size=voxel, truncation=3 * voxel, value_capacity=1 << 16, bucket_count=1 << 16,
                             max_vertex_count=1 << 18, max_triangle_count=1 << 18, **over)


class Images:
    """Device outputs of a raycast, started from a value no raycast writes."""

    def __init__(self, v):
        self.t = [torch.full((v.RH * v.RW * k,), 7.0, device="cuda") for k in (1, 4, 4)]

    def clear(self):
        for t in self.t:
            t.fill_(7.0)
        torch.cuda.synchronize()

    def host(self):
        torch.cuda.synchronize()
        return [t.cpu().numpy() for t in self.t]


def _same(images, expected):
    for got, want in zip(images.host(), expected):
        np.testing.assert_array_equal(got.view(np.uint32), np.asarray(want).reshape(-1).view(np.uint32))


def _capture(stream, call):
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=stream):
        call()
    return g


# cells of 2 voxels and of more, blocks from the dense array and (1 mm) from the hash table
@pytest.mark.parametrize("w,h,voxel", [(124, 92, 0.008), (52, 44, 0.0047), (40, 28, 0.001), (321, 203, 0.016)])
@pytest.mark.parametrize("first", [False, True])
def test_replayed_raycast(built, w, h, voxel, first):
    wl = scene.full_spline(6, width=w, height=h)
    stream = torch.cuda.Stream()
    v = Volume(_params(wl, voxel), stream=stream.cuda_stream)
    for k in range(6):
        v.integrate_frame(wl.frame(k), wl.pose(k))
    T = np.asarray(wl.pose(5), np.float64)
    poses = [T, left_update(T, [0.1, -0.07, 0.05, 0.1, 0.2, -0.15]), left_update(T, [3.0, -2.0, 0.4, 0.0, 0.0, 2.5]),
             T @ np.diag([1.2, 0.8, 1.1, 1.0]), left_update(T, [40.0, 40.0, 0.0, 0.0, 0.0, 0.0])]
    out = Images(v)
    if not first:                        # else the grid's memory is taken in the capture
        v.raycast(_cTw(T))
    g = _capture(stream, lambda: v.raycast(_cTw(poses[4]), *out.t))   # a view without the map
    hits = []
    pos, f = v.dump_blocks()
    for part in (slice(None), slice(0, None, 2), slice(1, None, 3)):
        if part != slice(None):
            # the map's blocks change, their places in the pool too
            v.reset()
            v.load_blocks(pos[part], f["sdf"][part], f["w"][part])
        for P in poses + poses[:1]:
            want = v.raycast(_cTw(P))    # the volume's pose from here on
            out.clear()
            g.replay()
            _same(out, want)
            g.replay()
            _same(out, want)
            hits.append(int(np.isfinite(want[0]).sum()))
    assert hits[0] > w * h // 4 and hits[4] == 0 and hits[0] == hits[5]
    assert v.stats()["error"] == 0


def test_replays_between_more_raycasts_than_tags(built):
    wl = scene.full_spline(6, width=36, height=28)
    stream = torch.cuda.Stream()
    v = Volume(_params(wl, 0.016), stream=stream.cuda_stream)
    for k in range(6):
        v.integrate_frame(wl.frame(k), wl.pose(k))
    pos, f = v.dump_blocks()
    T = np.asarray(wl.pose(5), np.float64)
    out = Images(v)
    full = v.raycast(_cTw(T))
    g = _capture(stream, lambda: v.raycast(_cTw(T), *out.t))
    for k in range(3):
        v.reset()
        v.load_blocks(pos[k::3], f["sdf"][k::3], f["w"][k::3])
        want = v.raycast(_cTw(T))
        for _ in range(101):
            for a, b in zip(v.raycast(_cTw(T)), want):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
        g.replay()
        _same(out, want)
    assert np.isfinite(full[0]).any()


@pytest.mark.parametrize("psdf", [False, True])
def test_replayed_frame(built, psdf):
    wl = scene.full_spline(12, width=96, height=72)
    stream = torch.cuda.Stream()
    p = _params(wl, 0.008, bayesian=psdf)
    v, u = Volume(p, stream=stream.cuda_stream), Volume(p, stream=stream.cuda_stream)
    for x in (v, u):
        for k in range(3):
            x.integrate_frame(wl.frame(k), wl.pose(k), tv_iterations=3)
        x.raycast(_cTw(wl.pose(2)))
    depth = torch.from_numpy(np.ascontiguousarray(wl.frame(3))).cuda()
    T = wl.pose(3)
    out, ref = Images(v), Images(u)

    def frame(x, images):
        x.integrate_frame(depth, T, on_device=True, tv_iterations=3, ray_depth=images.t[0], ray_vertex=images.t[1],
                          ray_normal=images.t[2], outputs_on_device=True)
    g = _capture(stream, lambda: frame(v, out))
    for k in range(4):
        depth.copy_(torch.from_numpy(np.ascontiguousarray(wl.frame(3 + k))))
        torch.cuda.synchronize()
        out.clear()
        g.replay()
        frame(u, ref)
        _same(out, ref.host())
    (pa, fa), (pb, fb) = v.dump_blocks(), u.dump_blocks()
    ia, ib = np.lexsort(pa.T), np.lexsort(pb.T)
    np.testing.assert_array_equal(pa[ia], pb[ib])
    for key in fa:
        np.testing.assert_array_equal(fa[key][ia].view(np.uint32), fb[key][ib].view(np.uint32))
    assert v.stats()["error"] == 0 and u.stats()["error"] == 0


def _same_blocks(v, u):
    (pa, fa), (pb, fb) = v.dump_blocks(), u.dump_blocks()
    ia, ib = np.lexsort(pa.T), np.lexsort(pb.T)
    np.testing.assert_array_equal(pa[ia], pb[ib])
    np.testing.assert_array_equal(fa["sdf"][ia].view(np.uint32), fb["sdf"][ib].view(np.uint32))
    return fa["sdf"][ia]


def _iterate(v, iterations):
    v._c("mh_huber_tv_iterate", 2.0, 8.0, 0.01, iterations, None, v.stream)   # no energies: nothing waits


@pytest.mark.parametrize("iterations", [1, 3])
def test_replayed_huber_tv(built, iterations):
    wl = scene.full_spline(6, width=96, height=72)
    stream = torch.cuda.Stream()
    p = _params(wl, 0.008)
    v = Volume(p, stream=stream.cuda_stream)
    for k in range(6):
        v.integrate_frame(wl.frame(k), wl.pose(k))
    v.collect_all_blocks()
    u = Volume(p, stream=stream.cuda_stream)
    pos, f = v.dump_blocks()
    u.load_blocks(pos, f["sdf"], f["w"])
    w = f["w"]
    seen = [f["sdf"]]

    def both(call):
        for x in (v, u):
            call(x)
    both(lambda x: x.set_candidates(pos))
    both(lambda x: x.huber_tv_init())
    g = _capture(stream, lambda: _iterate(v, iterations))

    def step():
        torch.cuda.synchronize()         # the replay is on another stream
        g.replay()
        torch.cuda.synchronize()
        _iterate(u, iterations)
        seen.append(_same_blocks(v, u))
        assert not np.array_equal(seen[-1], seen[-2])
    step()
    step()
    both(lambda x: _iterate(x, 2))       # the volume's own call in between
    step()
    # neighbours that are no candidates any more, then with other weights
    both(lambda x: x.set_candidates(pos[::2]))
    step()
    rng = np.random.default_rng(0)
    some = np.where(rng.random(w.shape) < 0.2, 0.0, w).astype(np.float32)
    both(lambda x: x.load_blocks(pos[1::2], None, some[1::2]))
    step()
    both(lambda x: x.set_candidates(pos[1::2]))
    step()
    # init and iterations in one graph
    both(lambda x: x.set_candidates(pos))
    h = _capture(stream, lambda: (v.huber_tv_init(), _iterate(v, iterations)))
    for own in (0, 1, 2):
        h.replay()
        torch.cuda.synchronize()
        u.huber_tv_init()
        _iterate(u, iterations)
        _same_blocks(v, u)
        both(lambda x: _iterate(x, own))
        _same_blocks(v, u)
    assert v.stats()["error"] == 0 and u.stats()["error"] == 0
