"""FP64 levels with few groups (each smoothed by a cluster) against the CPU oracle: V-cycles
bit for bit at one group and at the group counts where the cluster size changes, also with
no, one and several sweeps and relaxes; solves within the tolerance.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
import oracle as O
from femgpu import meshes

pytestmark = pytest.mark.gpu


# groups of level 0: 1, 9, about 19 | 20, 38 | 40, 76 | 80 (clusters of 8, 4, 2, 1)
@pytest.mark.parametrize("n,opts", [(18, {}), (64, {}), (92, {}), (97, {}), (133, {}), (140, {}), (188, {}), (200, {}),
                                    (40, dict(preInnerIters=0, postInnerIters=0)),
                                    (40, dict(preInnerIters=1, postInnerIters=1)), (40, dict(postRelaxes=3)),
                                    (40, dict(postRelaxes=0)), (40, dict(smootherWeight=0.7))])
def test_vcycle_matches_oracle(n, opts):
    xyz, conn = meshes.jittered_square(n)
    mask = meshes.boundary_mask_2d(n)
    kappa = np.ones(conn.shape[0])
    with femgpu.Solver(solverType=1, tolerance=1e-8, maxIters=600, flexibleCG=1, precision=1, **opts) as s:
        s.set_mesh(xyz, conn)
        s.assemble(kappa, 0.0)
        s.set_dirichlet(mask)
        s.setup()
        rp, ci, v = s.matrix()
        gx, ga = meshes.adjacency_from_pattern(rp, ci)
        names = dict(preInnerIters="pre_inner", postInnerIters="post_inner", postRelaxes="post_relaxes",
                     smootherWeight="smoother_weight")
        orc = O.OracleAMG(rp, ci, v, gx, ga, seed=1, fp64_hierarchy=1, **{names[k]: o for k, o in opts.items()})
        r = np.random.default_rng(1).standard_normal(xyz.shape[0])
        assert np.array_equal(s.vcycle(r), orc.vcycle(r))
        if not opts and n <= 64:
            x, st = s.solve(r)
            xo, sto = orc.pcg(r, tol=1e-8, max_iters=600, flexible=True)
            assert st["status"] == 0 and abs(st["iterations"] - sto["iters"]) <= 1
            assert np.linalg.norm(x - xo) / np.linalg.norm(xo) <= 1e-8
