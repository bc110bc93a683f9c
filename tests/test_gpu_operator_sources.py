"""One handle given meshes and matrices in turn: a mesh that is refused leaves no operator, an
assembly after a matrix is the mesh's own, and a matrix of the mesh's size is aggregated on the
mesh's graph whatever was set between.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
import oracle as O
from femgpu import meshes
from test_gpu_long_rows import arrow

pytestmark = pytest.mark.gpu

INVALID, NOT_READY = 1, 3


def status(call, *args):
    with pytest.raises(femgpu.FemgpuError) as e:
        call(*args)
    return e.value.status


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("vertex", [-1, 10 ** 6])
def test_a_refused_mesh_leaves_no_operator(dim, vertex):
    xyz, conn = meshes.kuhn_cube(3) if dim == 3 else meshes.jittered_square(6)
    bad = conn.copy()
    bad[5, 1] = vertex
    n = xyz.shape[0]
    with femgpu.Solver(solverType=1) as s:
        s.set_mesh(xyz, conn)
        s.assemble(None, 1.0)
        _, _, v = s.matrix()
        assert status(s.set_mesh, xyz, bad) == INVALID
        assert status(s.assemble, None, 1.0) == NOT_READY
        assert status(s.load_vector, np.ones(n)) == NOT_READY
        assert status(s.setup) == NOT_READY
        assert status(s.profile_kernel, 6, 1) == NOT_READY
        s.set_mesh(xyz, conn)
        s.assemble(None, 1.0)
        assert np.array_equal(s.matrix()[2], v)
        # arguments that are refused before anything is replaced leave the operator
        assert status(s.set_mesh, xyz[:0], conn) == INVALID
        assert np.array_equal(s.matrix()[2], v)


@pytest.mark.parametrize("other", ["same size", "smaller", "larger"])
def test_assembly_after_a_matrix_is_the_mesh_operator(other):
    xyz, conn = meshes.kuhn_cube(4)
    n = xyz.shape[0]
    rp, ci = O.build_pattern(n, conn)
    v = O.assemble(xyz, conn, rp, ci, coef=None, lambda_mass=1.0)
    with femgpu.Solver() as s:
        s.set_mesh(xyz, conn)
        m = {"same size": n, "smaller": n // 2, "larger": 3 * n}[other]
        s.set_matrix_csr(*arrow(m))  # one row of m entries, past the row gather's 32
        assert s.matrix()[0].shape[0] == m + 1
        for _ in range(2):
            s.assemble(None, 1.0)
            grp, gci, gv = s.matrix()
            assert np.array_equal(grp, rp) and np.array_equal(gci, ci) and np.array_equal(gv, v)


def test_matrix_of_the_mesh_size_keeps_the_mesh_graph():
    xyz, conn, kappa, f, mask = meshes.poisson3d_problem(9, sigma=1.0)
    n = xyz.shape[0]
    rp, ci = O.build_pattern(n, conn)
    v = O.assemble(xyz, conn, rp, ci, coef=kappa, lambda_mass=1.0)
    r = np.random.default_rng(0).standard_normal(n)
    out = []
    for between in (False, True):
        with femgpu.Solver(solverType=1, seed=1) as s:
            s.set_mesh(xyz, conn)
            if between:
                s.set_matrix_csr(*arrow(n // 3))
            s.set_matrix_csr(rp, ci, v)
            s.setup()
            out.append((s.num_levels, s.level(0)["perm"], s.vcycle(r)))
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
