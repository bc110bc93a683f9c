"""A caller's memory pool (femgpu_config.mem_pool) holds no more of a handle's memory than the
handle's live buffers: what a call frees is back in the pool when the call returns.  Needs a
GB300."""
import ctypes as C

import numpy as np
import pytest

import femgpu
from femgpu import meshes
from test_gpu_failures import _CappedPool

pytestmark = pytest.mark.gpu

_USED_MEM_CURRENT = 7  # CUmemPool_attribute, cuda.h


def used(pool):
    v = C.c_uint64()
    assert pool.cu.cuMemPoolGetAttribute(pool.pool, _USED_MEM_CURRENT, C.byref(v)) == 0
    return v.value


@pytest.fixture
def pool():
    torch = pytest.importorskip("torch")
    torch.cuda.init()
    femgpu.Solver().close()  # the runtime has a current context for the driver calls
    p = _CappedPool(256 << 20)
    yield p
    p.close()


@pytest.mark.parametrize("dim,n", [(2, 30), (3, 6), (3, 12)])
def test_freed_buffers_are_back_in_the_pool(pool, dim, n):
    import torch

    xyz, conn = meshes.jittered_square(n) if dim == 2 else meshes.kuhn_cube(n)
    nv, ne, k = xyz.shape[0], conn.shape[0], dim + 1
    s = femgpu.Solver(mem_pool=pool.pool.value)
    s.set_mesh(xyz, conn)
    s.assemble(np.ones(ne), 1.0)
    torch.cuda.synchronize()
    rp, ci, _ = s.matrix()
    nnz = ci.shape[0]
    # mesh, incidence lists, slot map, operator, aggregation graph, coefficients
    live = [24 * nv, 4 * k * ne, 4 * (nv + 1), 4 * k * ne, k * k * ne, 4 * (nv + 1), 4 * nnz, 8 * nnz, 4 * (nv + 1),
            4 * (nnz - nv), 8 * ne]
    assert sum(live) <= used(pool) <= sum((b + 511) // 512 * 512 for b in live)
    before = used(pool)
    for _ in range(2):
        s.load_vector(np.ones(nv))
        assert used(pool) == before
    s.close()
    assert used(pool) == 0


def test_setup_and_solve_on_a_caller_pool_keep_their_bits(pool):
    xyz, conn, kappa, f, mask = meshes.poisson3d_problem(10, sigma=1.0)
    out = []
    for mem_pool in (None, pool.pool.value):
        with femgpu.Solver(solverType=1, tolerance=1e-8, maxIters=200, flexibleCG=1, seed=1, mem_pool=mem_pool) as s:
            s.set_mesh(xyz, conn)
            s.assemble(kappa, 0.0)
            s.set_dirichlet(mask)
            b = np.where(mask.astype(bool), 0.0, s.load_vector(f))
            for _ in range(2):
                s.setup()
                x, st = s.solve(b)
                assert st["status"] == 0
                out.append(x)
    assert all(np.array_equal(x, out[0]) for x in out)
