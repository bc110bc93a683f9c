"""An operator with one row past the sorting tiers' capacity (8192 entries), whose permuted row
takes the dense accumulator: column counts on both sides of the 48 KB that a kernel may use
without asking (accumulator, marks and the kernel's own arrays).  Levels bit for bit against the
CPU oracle, and the solution.  Needs a GB300."""
import numpy as np
import pytest
import scipy.sparse as sp

import femgpu
import oracle as O
from femgpu import meshes

pytestmark = pytest.mark.gpu


def arrow(n):
    """A hub coupled to every other row."""
    i = np.arange(1, n)
    w = np.random.default_rng(n).uniform(0.5, 1.0, n - 1) / n
    rows, cols = np.r_[np.arange(n), 0 * i, i], np.r_[np.arange(n), i, 0 * i]
    A = sp.coo_matrix((np.r_[np.linspace(2.0, 4.0, n), -w, -w], (rows, cols)), shape=(n, n)).tocsr()
    A.sort_indices()
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data


@pytest.mark.parametrize("n", [8193, 9804, 9805, 9830, 9831])
def test_dense_row_at_the_shared_memory_limit(n):
    rp, ci, v = arrow(n)
    orc = O.OracleAMG(rp, ci, v, *meshes.adjacency_from_pattern(rp, ci), seed=1, partition_max=n)
    b = np.random.default_rng(1).uniform(-1.0, 1.0, n)
    with femgpu.Solver(solverType=1, tolerance=1e-10, maxIters=50, flexibleCG=1, seed=1, partitionMaxSize=n) as s:
        s.set_matrix_csr(rp, ci, v)
        s.setup()
        assert s.num_levels == orc.num_levels == 2
        for l in range(2):
            go, oo = s.level(l), orc.level(l)
            for key in ("A_rowptr", "A_cols", "A_vals"):
                assert np.array_equal(go[key], oo[key]), (l, key)
        for key in ("perm", "agg_idx", "part_idx", "P_rowptr", "P_cols", "P_vals"):
            assert np.array_equal(s.level(0)[key], orc.level(0)[key]), key
        x, st = s.solve(b)
    assert st["status"] == 0
    A = sp.csr_matrix((v, ci, rp))
    assert np.linalg.norm(A @ x - b) <= 2e-10 * np.linalg.norm(b)
