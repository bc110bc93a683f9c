"""One handle given meshes in turn: a mesh that is refused leaves no operator.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
from femgpu import meshes

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
