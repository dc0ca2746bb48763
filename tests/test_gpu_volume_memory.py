"""The memory of the view's grid comes with the first raycast, where it is not a
small part of the volume's.

Two volumes that differ in the raycast's depth only: the farther view's grid is
larger by tens of megabytes, which a volume takes when it casts rays, not before,
and once.
"""
import numpy as np
import pytest

from meshhashing_gb300 import Batch, Volume, config, scene

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MB = 1 << 20


def _taken(call):
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    out = call()
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0], out


def _params(depth):
    wl = scene.full_spline(4)
    p = config.params_for(wl, value_capacity=1 << 13, bucket_count=1 << 13, max_vertex_count=1 << 14,
                          max_triangle_count=1 << 14, mesh_page_capacity=1 << 10)
    p.max_raycast_depth = depth
    return wl, p


def test_first_raycast_takes_the_grid(built):
    wl, near = _params(1.0)
    _, far = _params(5.5)
    cTw = np.linalg.inv(np.asarray(wl.pose(0), np.float64)).astype(np.float32)
    first, _ = _taken(lambda: Volume(near))       # the library's own start is paid here
    a, v = _taken(lambda: Volume(near))
    b, u = _taken(lambda: Volume(far))
    assert abs(a - b) <= 4 * MB
    c, _ = _taken(lambda: v.raycast(cTw))
    d, _ = _taken(lambda: u.raycast(cTw))
    e, _ = _taken(lambda: u.raycast(cTw))
    assert d - c > 40 * MB and e <= 2 * MB
    w = Volume(far)
    g, batch = _taken(lambda: Batch([w], raycast=True))
    assert g > 40 * MB
    h, _ = _taken(lambda: batch.step([np.full((480, 640), 1.0, np.float32)], [wl.pose(0)]))
    assert h <= 16 * MB                           # but the kernels' code on its first launch
    batch.close()
