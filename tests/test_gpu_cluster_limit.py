"""Setup on a device that runs smaller thread-block clusters, or none: the aggregation in fewer
CTAs and the coarsest factorisation in one block, bit for bit against the CPU oracle.  Needs a
GB300 (the limit is lowered on the handle)."""
import numpy as np
import pytest

import femgpu
import oracle as O
from femgpu import meshes
from test_gpu_coarsest import dense_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [1, 8, 33, 129, 392])
@pytest.mark.parametrize("limit", [1, 7])
def test_inverse_without_the_cluster(n, limit, precision):
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n)) * (rng.random((n, n)) < 0.6)
    M[np.arange(n), (np.arange(n) + 1) % n] += 3.0 * n
    rp, ci, v = dense_csr(M)
    orc = O.OracleAMG(rp, ci, v, *meshes.adjacency_from_pattern(rp, ci), max_levels=1, top_size=1,
                      fp64_hierarchy=precision)
    with femgpu.Solver(solverType=0, maxLevels=1, topSize=1, precision=precision) as s:
        s.test_cluster_limit(limit)
        s.set_matrix_csr(rp, ci, v)
        s.setup()
        for k in (0, n // 2, n - 1):
            r = np.zeros(n)
            r[k] = 1.0
            assert np.array_equal(s.vcycle(r), orc.vcycle(r))


def test_singular_without_the_cluster():
    M = np.eye(40)
    M[:, 17], M[17, 18] = 0.0, 1.0
    with femgpu.Solver(solverType=0, maxLevels=1, topSize=1) as s:
        s.test_cluster_limit(1)
        s.set_matrix_csr(*dense_csr(M))
        with pytest.raises(femgpu.FemgpuError) as e:
            s.setup()
        assert e.value.status == 4  # FEMGPU_ERR_BREAKDOWN


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("limit", [1, 2, 8, 0])
def test_hierarchy_in_smaller_clusters(limit, precision):
    xyz, conn, kappa, f, mask = meshes.poisson3d_problem(17, sigma=1.0)
    rp, ci = O.build_pattern(xyz.shape[0], conn)
    v = O.assemble(xyz, conn, rp, ci, coef=kappa, lambda_mass=0.0)
    v, _ = O.apply_dirichlet(rp, ci, v, mask, None)
    orc = O.OracleAMG(rp, ci, v, *meshes.adjacency_from_pattern(rp, ci), seed=1, fp64_hierarchy=precision)
    with femgpu.Solver(solverType=1, seed=1, precision=precision) as s:
        s.test_cluster_limit(limit)
        s.set_mesh(xyz, conn)
        s.assemble(kappa, 0.0)
        s.set_dirichlet(mask)
        s.setup()
        assert s.num_levels == orc.num_levels >= 2
        for l in range(orc.num_levels):
            go, oo = s.level(l), orc.level(l)
            keys = ["A_rowptr", "A_cols", "A_vals"] + (["perm", "agg_idx", "part_idx"] if oo["n_agg"] else [])
            for key in keys:
                assert np.array_equal(go[key], oo[key]), (l, key)
        r = np.random.default_rng(2).standard_normal(xyz.shape[0])
        z = s.vcycle(r)
    with femgpu.Solver(solverType=1, seed=1, precision=precision) as s:  # the coarsest inverse included
        s.set_mesh(xyz, conn)
        s.assemble(kappa, 0.0)
        s.set_dirichlet(mask)
        s.setup()
        assert np.array_equal(z, s.vcycle(r))
