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


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("half", [2, 7, 8, 31, 32, 63, 64, 100])
def test_banded_hierarchies(half, precision):
    # rows of 5, 15, 17, 63, 65, 127, 129 and 201 entries: the row tiers of the permuted operator
    # and the prolongator (16, 64, 128, 256), products with and without direct slots
    n = 4000
    rng = np.random.default_rng(half)
    i = np.arange(n)
    lo, hi = np.maximum(0, i - half), np.minimum(n, i + half + 1)
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(hi - lo, out=rp[1:])
    rows = np.repeat(i, hi - lo)
    ci = (np.arange(rp[-1]) - np.repeat(rp[:-1], hi - lo) + np.repeat(lo, hi - lo)).astype(np.int32)
    w = rng.uniform(0.5, 1.0, (n, half + 1))
    v = np.where(ci == rows, 0.0, -w[np.minimum(rows, ci), np.abs(rows - ci)])
    v[ci == rows] = 1.0 - np.bincount(rows, weights=v, minlength=n)
    gx, ga = meshes.adjacency_from_pattern(rp, ci)
    part = 512 if 7 <= half < 60 else 1024
    orc = O.OracleAMG(rp, ci, v, gx, ga, seed=1, fp64_hierarchy=precision, max_levels=2, partition_max=part)
    with femgpu.Solver(precision=precision, maxLevels=2, partitionMaxSize=part) as s:
        s.set_matrix_csr(rp, ci, v)
        s.setup()
        assert s.num_levels == orc.num_levels
        for l in range(orc.num_levels):
            got, want = s.level(l), orc.level(l)
            for key in want:
                assert np.array_equal(got[key], want[key]), (l, key)
        r = rng.standard_normal(n)
        assert np.array_equal(s.vcycle(r), orc.vcycle(r))
