"""Meshes with many vertices of high degree numbered together: their candidate lists pass the
warp's (1024) and the block's (8192) sorting capacity side by side, in blocks of the long-segment
kernel that hold none, one or several of them.  Pattern against the CPU oracle.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
import oracle as O

pytestmark = pytest.mark.gpu


def fans(sizes):
    """A fan of sizes[h] triangles around vertex h for every h, each with its own ring."""
    hubs = len(sizes)
    start = hubs + np.concatenate([[0], np.cumsum(sizes)])
    xyz = np.random.default_rng(hubs).uniform(-1.0, 1.0, (start[-1], 3))
    xyz[:, 2] = 0.0
    conn = [np.stack([np.full(k, h), start[h] + np.arange(k), start[h] + (np.arange(k) + 1) % k], axis=1)
            for h, k in enumerate(sizes)]
    return xyz, np.concatenate(conn).astype(np.int32)


@pytest.mark.parametrize("hubs,long_from", [(1, 0), (7, 3), (304, 290), (305, 0), (1024, 1000), (2000, 1300)])
def test_pattern_with_neighbouring_hubs(hubs, long_from):
    rng = np.random.default_rng(hubs)
    sizes = rng.integers(3, 12, hubs)
    longs = rng.random(hubs) < 0.9
    longs[:long_from] = False
    longs[-1] = True
    sizes[longs] = rng.integers(342, 420, int(longs.sum()))  # 3 candidates per triangle
    sizes[-1] = 2731
    xyz, conn = fans(sizes)
    rp, ci = O.build_pattern(xyz.shape[0], conn)
    with femgpu.Solver() as s:
        s.set_mesh(xyz, conn)
        s.assemble(None, 1.0)
        grp, gci, _ = s.matrix()
    assert np.array_equal(grp, rp) and np.array_equal(gci, ci)
