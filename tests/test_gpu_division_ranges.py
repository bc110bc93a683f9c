"""The hand-written divisions at the ends of their operand windows, bit for bit against the CPU
oracle, which divides: the coarsest inverse (reciprocal with two corrections between 2^-511 and
2^511, not for divisors of an all-ones significand, zeros by themselves) on scaled matrices, and
the assembly's constant divisions (|x| between 2^-975 and 2^977) on scaled meshes.  Needs a
GB300."""
import numpy as np
import pytest

import femgpu
import oracle as O
from femgpu import meshes
from test_gpu_coarsest import dense_csr

pytestmark = pytest.mark.gpu


def inverse_matches(M):
    n = M.shape[0]
    rp, ci, v = dense_csr(M)
    orc = O.OracleAMG(rp, ci, v, *meshes.adjacency_from_pattern(rp, ci), max_levels=1, top_size=1, fp64_hierarchy=1)
    with femgpu.Solver(solverType=0, maxLevels=1, topSize=1, precision=1) as s:
        s.set_matrix_csr(rp, ci, v)
        s.setup()
        for k in range(0, n, max(1, n // 5)):
            r = np.zeros(n)
            r[k] = 1.0
            assert np.array_equal(s.vcycle(r), orc.vcycle(r), equal_nan=True), k


@pytest.mark.parametrize("n", [9, 40, 130])
@pytest.mark.parametrize("exponent", [-1010, -513, -512, -511, -510, 0, 508, 509, 510, 511, 512, 900])
def test_scaled_matrix(n, exponent):
    # pivots from just below to just above 2^exponent
    rng = np.random.default_rng(n + exponent + 2000)
    M = np.triu(rng.uniform(-0.5, 0.5, (n, n)) * (rng.random((n, n)) < 0.5), 1)
    M += np.diag(rng.uniform(0.5, 2.0, n)) + np.tril(rng.uniform(-0.1, 0.1, (n, n)), -1)
    inverse_matches(np.ldexp(M, exponent))


@pytest.mark.parametrize("n", [9, 40, 130])
@pytest.mark.parametrize("spread", [40, 260, 520])
def test_rows_and_columns_of_different_scales(n, spread):
    # numerators and divisors of every exponent, quotients that leave the normal range
    rng = np.random.default_rng(n + spread)
    M = rng.uniform(-1.0, 1.0, (n, n)) * (rng.random((n, n)) < 0.3) + np.diag(rng.uniform(4.0, 8.0, n))
    e = rng.integers(-spread, spread + 1, n)
    M = np.ldexp(M, e[:, None] + rng.permutation(e)[None] // 2)
    inverse_matches(np.where(M == 0.0, 0.0, M))


@pytest.mark.parametrize("n", [9, 40, 130])
@pytest.mark.parametrize("steps", [1, 2, 0, -1])
def test_divisors_of_almost_all_ones(n, steps):
    # upper triangular: the pivots are the diagonal, `steps` units below a power of two
    rng = np.random.default_rng(n)
    d = np.ldexp(1.0, rng.integers(-30, 31, n))
    d = d * (1.0 - steps * 2.0 ** -53) if steps >= 0 else d * (1.0 + 2.0 ** -52)
    M = np.triu(rng.uniform(-1.0, 1.0, (n, n)) * (rng.random((n, n)) < 0.4), 1) * np.abs(d)[:, None] + np.diag(d)
    inverse_matches(M)


@pytest.mark.parametrize("mass", [0.0, 1.0])
@pytest.mark.parametrize("dim,exponent", [(3, e) for e in (-340, -326, -325, -324, -320, 320, 324, 325, 326)] +
                         [(2, e) for e in (-530, -489, -488, -487, -486, -480, 486, 487, 488, 489, 490)])
def test_scaled_mesh(dim, exponent, mass):
    xyz, conn = meshes.kuhn_cube(3) if dim == 3 else meshes.jittered_square(7)
    rng = np.random.default_rng(exponent + 1000)
    xyz = xyz + rng.uniform(-0.05, 0.05, xyz.shape) * (np.arange(3) < dim)
    xyz = np.ldexp(xyz * 3.0, exponent)
    f = rng.uniform(-1.0, 1.0, xyz.shape[0])
    rp, ci = O.build_pattern(xyz.shape[0], conn)
    with femgpu.Solver() as s:
        s.set_mesh(xyz, conn)
        s.assemble(None, mass)
        v, b = s.matrix()[2], s.load_vector(f)
    assert np.array_equal(v, O.assemble(xyz, conn, rp, ci, coef=None, lambda_mass=mass), equal_nan=True)
    assert np.array_equal(b, O.load_vector(xyz, conn, f), equal_nan=True)
