"""The check of the blocks' masks finds a mask that hides a voxel."""
import numpy as np

from tests._neg_masks import GROUP, hidden, needed


def test_each_voxel_has_its_bit():
    for v in range(512):
        x, y, z = v % 8, v // 8 % 8, v // 64
        for value in (-1e-30, -1.0, np.nan, np.inf, 1e30):
            sdf = np.zeros((1, 512), np.float32)
            sdf[0, v] = value
            want = np.uint64(1) << np.uint64(x // 2 + 4 * (y // 2) + 16 * (z // 2))
            assert needed(sdf)[0] == want
    assert needed(np.array([[-0.0] * 512, [9e29] * 512], np.float32)).tolist() == [0, 0]


def test_a_missing_bit_is_found():
    rng = np.random.default_rng(0)
    sdf = np.where(rng.random((200, 512)) < 0.02, -1.0, 1.0).astype(np.float32)
    mask = needed(sdf)
    assert hidden(sdf, mask).size == 0
    assert hidden(sdf, np.full(200, 2 ** 64 - 1, np.uint64)).size == 0   # bits without need
    for b in range(200):
        v = int(np.argmax(sdf[b] < 0))
        if sdf[b, v] < 0:
            planted = mask.copy()
            planted[b] &= ~(np.uint64(1) << np.uint64(GROUP[v]))
            assert hidden(sdf, planted).tolist() == [b]
