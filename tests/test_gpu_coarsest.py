"""The coarsest level's explicit inverse against the CPU oracle, bit for bit, at the sizes
where its kernels change shape (panels of 8, warps of 32, registers per lane, the largest
matrix that stays on chip), with row exchanges; and a singular matrix.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
import oracle as O
from femgpu import meshes

pytestmark = pytest.mark.gpu


def dense_csr(M):
    n = M.shape[0]
    keep = M != 0
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(keep.sum(axis=1), out=rp[1:])
    return rp, np.nonzero(keep)[1].astype(np.int32), M[keep]


def pair(M, precision):
    """(solver, oracle hierarchy) whose only level is M's dense factorisation."""
    rp, ci, v = dense_csr(M)
    gx, ga = meshes.adjacency_from_pattern(rp, ci)
    s = femgpu.Solver(solverType=0, maxLevels=1, topSize=1, precision=precision)
    s.set_matrix_csr(rp, ci, v)
    return s, O.OracleAMG(rp, ci, v, gx, ga, max_levels=1, top_size=1, fp64_hierarchy=precision)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 150, 200, 256, 257, 384, 391, 392, 393])
def test_inverse_matches_oracle(n, precision):
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n)) * (rng.random((n, n)) < 0.6)  # no dominant diagonal: rows are exchanged
    M[np.arange(n), (np.arange(n) + 1) % n] += 3.0 * n
    s, orc = pair(M, precision)
    s.setup()
    for k in (0, n // 2, n - 1):
        r = np.zeros(n)
        r[k] = 1.0
        assert np.array_equal(s.vcycle(r), orc.vcycle(r))
    s.close()


@pytest.mark.parametrize("n,zero", [(5, 0), (40, 17), (130, 129), (393, 300)])
def test_singular_matrix_is_a_breakdown(n, zero):
    M = np.eye(n) + np.diag(np.full(n - 1, 0.25), 1)
    M[:, zero] = 0.0
    M[zero, (zero + 1) % n] = 1.0  # no empty row
    rp, ci, v = dense_csr(M)
    with femgpu.Solver(solverType=0, maxLevels=1, topSize=1) as s:
        s.set_matrix_csr(rp, ci, v)
        with pytest.raises(femgpu.FemgpuError) as e:
            s.setup()
        assert e.value.status == 4  # FEMGPU_ERR_BREAKDOWN
        s.set_matrix_csr(*dense_csr(np.eye(n) * 2.0))
        s.setup()
        assert np.array_equal(s.vcycle(np.ones(n)), np.full(n, 0.5))
