"""The rule of a block's mask, shared by its CPU and GPU tests."""
import numpy as np

_V = np.arange(512)
GROUP = (_V & 7) // 2 + 4 * ((_V >> 3 & 7) // 2) + 16 * ((_V >> 6) // 2)   # of each voxel


def needed(sdf):
    """Masks (uint64 per block) with the bits that have to be set: those of the
    voxels whose sdf does not lie in [0, 1e30)."""
    sdf = np.asarray(sdf, np.float32)
    with np.errstate(invalid="ignore"):
        out = ~((sdf >= np.float32(0.0)) & (sdf < np.float32(1e30)))
    bits = np.zeros((len(sdf), 64), bool)
    for g in range(64):
        bits[:, g] = out[:, GROUP == g].any(axis=1)
    return (bits.astype(np.uint64) << np.arange(64, dtype=np.uint64)).sum(axis=1, dtype=np.uint64)


def hidden(sdf, mask):
    """Blocks of which the mask hides a voxel: a clear bit over one that needs it."""
    return np.nonzero(needed(sdf) & ~np.asarray(mask, np.uint64))[0]
