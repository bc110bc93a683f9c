"""The block solve's smoother paths against single-column solves: all eight columns per CTA
(at least 304 groups), split columns, groups past 512 rows, other post relax counts, in both
precisions.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
from femgpu import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n,opts", [(51, {}), (20, {}), (16, dict(partitionMaxSize=900)), (12, dict(postRelaxes=0)),
                                    (12, dict(postRelaxes=2)), (12, dict(preInnerIters=1, postInnerIters=4))])
def test_columns_match_single_solves(n, opts, precision):
    xyz, conn, kappa, _, mask = meshes.poisson3d_problem(n, sigma=1.0)
    with femgpu.Solver(solverType=1, tolerance=1e-8, maxIters=600, flexibleCG=1, seed=2, precision=precision,
                       **opts) as s:
        s.set_mesh(xyz, conn)
        s.assemble(kappa, 0.0)
        s.set_dirichlet(mask)
        rng = np.random.default_rng(n)
        B = np.where(mask.astype(bool)[:, None], 0.0, rng.uniform(-1.0, 1.0, (xyz.shape[0], 10)))
        s.setup()
        X, st = s.solve_multi(B)
        assert st["status"] == 0 and st["relres"] <= 1e-8
        for j in (0, 5, 7, 9):
            x, _ = s.solve(B[:, j])
            # both are within the tolerance of A x = b from the same iteration: the FP32 V-cycle's
            # rounding moves an iterate by far less than its distance from the solution
            assert np.linalg.norm(X[:, j] - x) / np.linalg.norm(x) <= 1e-8, j
