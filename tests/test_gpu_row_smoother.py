"""The row smoother (levels with many groups and rows of more than 16 in-partition entries)
against the CPU oracle: hierarchies and V-cycles bit for bit, on banded operators with rows of
uneven length, at 2 to 16 sums per row, in FP32 and over clusters of 4, 2 and 1 CTAs in FP64,
with no, one and several sweeps.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
import oracle as O
from femgpu import meshes

pytestmark = pytest.mark.gpu


def banded(n, half, keep, far=0):
    """SPD operator: a random part of the band |i - j| <= half, every 37th row and column out
    to `far` as well."""
    rng = np.random.default_rng(half + n)
    reach = max(half, far)
    i = np.repeat(np.arange(n), reach)
    d = np.tile(np.arange(1, reach + 1), n)
    j = i + d
    in_band = (d <= half) & ((rng.random(i.size) < keep) | (d == 1))
    ok = (j < n) & (in_band | ((d <= far) & ((i % 37 == 0) | (j % 37 == 0))))
    i, j = i[ok], j[ok]
    w = -rng.uniform(0.5, 1.0, i.size)
    r, c, v = np.concatenate([i, j]), np.concatenate([j, i]), np.concatenate([w, w])
    diag = 1.0 - np.bincount(r, weights=v, minlength=n)
    r, c, v = np.concatenate([r, np.arange(n)]), np.concatenate([c, np.arange(n)]), np.concatenate([v, diag])
    order = np.lexsort((c, r))
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    return rp, c[order].astype(np.int32), v[order]


CASES = [
    # rows, half band, kept part of it, far rows, precision, groups at least, options
    (16000, 7, 0.7, 12, 0, 153, {}),  # 2 sums per row
    (18000, 9, 0.9, 0, 0, 153, {}),   # 4
    (17000, 17, 0.9, 0, 0, 77, {}),   # 8
    (12000, 34, 0.9, 0, 0, 26, {}),   # 16
    (6500, 17, 0.9, 0, 1, 26, {}),    # FP64, clusters of 4
    (9000, 17, 0.9, 0, 1, 39, {}),    # 2
    (18000, 17, 0.9, 0, 1, 77, {}),   # 1
    (11000, 34, 0.9, 0, 1, 26, {}),
    (17000, 17, 0.8, 0, 0, 77, dict(preInnerIters=0, postInnerIters=0)),
    (17000, 17, 0.8, 0, 0, 77, dict(preInnerIters=1, postInnerIters=2, postRelaxes=2)),
    (5600, 17, 0.8, 0, 1, 26, dict(preInnerIters=0, postInnerIters=1)),
    (17000, 17, 0.8, 0, 0, 77, dict(smootherWeight=0.7)),
]


@pytest.mark.parametrize("n,half,keep,far,precision,groups,opts", CASES)
def test_vcycle_matches_oracle(n, half, keep, far, precision, groups, opts):
    rp, ci, v = banded(n, half, keep, far)
    gx, ga = meshes.adjacency_from_pattern(rp, ci)
    names = dict(preInnerIters="pre_inner", postInnerIters="post_inner", postRelaxes="post_relaxes",
                 smootherWeight="smoother_weight")
    orc = O.OracleAMG(rp, ci, v, gx, ga, seed=1, fp64_hierarchy=precision, max_levels=2,
                      **{names[k]: o for k, o in opts.items()})
    with femgpu.Solver(precision=precision, maxLevels=2, **opts) as s:
        s.set_matrix_csr(rp, ci, v)
        s.setup()
        top = s.level(0)
        rows = np.diff(top["agg_idx"][top["part_idx"]]).max()  # no group is larger
        assert -(-n // rows) >= groups and rows <= 512
        r = np.random.default_rng(1).standard_normal(n)
        assert np.array_equal(s.vcycle(r), orc.vcycle(r))


@pytest.mark.parametrize("precision", [0, 1])
def test_copy_wait_running_out_reports_limit_and_handle_recovers(precision):
    rp, ci, v = banded(17000, 17, 0.9)
    r = np.random.default_rng(2).standard_normal(17000)
    with femgpu.Solver(solverType=1, precision=precision, maxLevels=2) as s:
        s.set_matrix_csr(rp, ci, v)
        s.setup()
        want, st = s.solve(r)
        assert st["status"] == 0
        s.test_copy_wait_limit(0)
        with pytest.raises(femgpu.FemgpuError) as e:
            s.vcycle(r)
        assert e.value.status == 6  # FEMGPU_ERR_LIMIT
        assert s.solve(r, check=False)[1]["status"] == 6
        s.test_copy_wait_limit(-1)
        assert np.array_equal(s.solve(r)[0], want)


@pytest.mark.parametrize("precision", [0, 1])
def test_saved_hierarchy_runs_the_same(tmp_path, precision):
    rp, ci, v = banded(17000, 17, 0.9)
    r = np.random.default_rng(3).standard_normal(17000)
    path = str(tmp_path / "h.bin")
    with femgpu.Solver(precision=precision, maxLevels=2) as s, femgpu.Solver(precision=precision, maxLevels=2) as t:
        s.set_matrix_csr(rp, ci, v)
        s.setup()
        s.save_hierarchy(path)
        t.set_matrix_csr(rp, ci, v)
        t.load_hierarchy(path)
        assert np.array_equal(s.vcycle(r), t.vcycle(r))
