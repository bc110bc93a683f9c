"""Aggregates, partitions and the next graph of small levels against the CPU oracle, bit for
bit, where the one-kernel aggregation changes shape: one to sixteen CTAs, last chunks of every
remainder, both sides of its size limit, partitions that must give nodes away, and other
distances and minimum sizes.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
import oracle as O
from femgpu import meshes

pytestmark = pytest.mark.gpu


def check(xyz, conn, **opts):
    rp, ci = O.build_pattern(xyz.shape[0], conn)
    gx, ga = meshes.adjacency_from_pattern(rp, ci)
    want = O.oldmis(gx, ga, params=opts.get("randMisParameters", 90102),
                    part_max=opts.get("partitionMaxSize", 512), seed=opts.get("seed", 1))
    with femgpu.Solver(topSize=256 if xyz.shape[0] > 256 else 32, **opts) as s:
        s.set_mesh(xyz, conn)
        s.assemble(None, 1.0)
        s.setup()
        got = s.level(0)
    for key in ("perm", "agg_idx", "part_idx"):
        assert np.array_equal(got[key], want[key]), key


# vertices: 64, 1024, 1089, 2116, 4096, 8281, 16641, 49284, 98596; edges at 315 and 316: 596,610
# and 600,400 (both sides of the limit of 600,000)
@pytest.mark.parametrize("n", [7, 31, 32, 45, 63, 90, 128, 221, 313, 315, 316])
def test_square_sizes(n):
    check(*meshes.jittered_square(n))


@pytest.mark.parametrize("n,opts", [
    (9, dict(partitionMaxSize=450, seed=7)), (9, dict(randMisParameters=50102)), (9, dict(randMisParameters=90202)),
    (9, dict(randMisParameters=90101, seed=3)), (9, dict(randMisParameters=10103)), (21, dict(partitionMaxSize=400)),
    (21, dict(partitionMaxSize=450, seed=7)), (21, dict(randMisParameters=50102))])
def test_cube_options(n, opts):
    check(*meshes.kuhn_cube(n), **opts)
