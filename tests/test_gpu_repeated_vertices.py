"""Elements that name a vertex more than once (collapsed elements of a mesh file), against a
sequential loop over the elements' whole matrices bit for bit, and twice: each pair of a
tetrahedron's and of a triangle's vertices, three and four equal vertices, on rows of the slot
map and past its limit.  The element matrices are the CPU oracle's, of the same coordinates under
distinct vertex numbers.  Needs a GB300; the first test shows on the CPU that such entries are
finite."""
import itertools

import numpy as np
import pytest

import femgpu
import oracle as O
from femgpu import meshes

GROUPS = {2: [(0, 1), (0, 2), (1, 2), (0, 1, 2)],
          3: list(itertools.combinations(range(4), 2)) + [(0, 2, 3), (1, 2, 3), (0, 1, 2, 3)]}


def collapsed(dim, group, hub=0):
    """A mesh on which every seventh element's vertices of `group` are its first one; hub: that
    many more elements around vertex 0, whose row then passes the slot map's 32 entries."""
    xyz, conn = meshes.kuhn_cube(4) if dim == 3 else meshes.jittered_square(9)
    rng = np.random.default_rng(5)
    xyz, conn = xyz + rng.uniform(-0.02, 0.02, xyz.shape) * (np.arange(3) < dim), conn.copy()
    if hub:
        fan = rng.permutation(xyz.shape[0] - 1)[:hub * dim].reshape(hub, dim) + 1
        conn = np.concatenate([conn, np.concatenate([np.zeros((hub, 1), np.int64), fan], axis=1)])
    conn[::7, list(group)] = conn[::7, group[0]:group[0] + 1]
    return xyz, np.ascontiguousarray(conn, dtype=np.int32)


def sequential(xyz, conn, coef, mass):
    rp, ci = O.build_pattern(xyz.shape[0], conn)
    k = conn.shape[1]
    own = np.arange(k, dtype=np.int32)[None]
    orp, oci = O.build_pattern(k, own)
    v = np.zeros(ci.shape[0])
    with np.errstate(all="ignore"):
        for e, ids in enumerate(conn):
            M = O.assemble(xyz[ids], own, orp, oci, coef=None if coef is None else coef[e:e + 1], lambda_mass=mass)
            for a in range(k):
                row = ci[rp[ids[a]]:rp[ids[a] + 1]]
                for b in range(k):
                    v[rp[ids[a]] + np.searchsorted(row, ids[b])] += M[a * k + b]
    return rp, ci, v


@pytest.mark.parametrize("dim,group", [(3, (1, 2)), (3, (1, 3)), (3, (2, 3)), (2, (0, 2)), (2, (1, 2))])
def test_entries_of_collapsed_elements_can_be_finite(dim, group):
    xyz, conn = collapsed(dim, group)
    own = np.arange(dim + 1, dtype=np.int32)[None]
    rp, ci = O.build_pattern(dim + 1, own)
    finite = 0
    for ids in conn[::7]:
        M = O.assemble(xyz[ids], own, rp, ci, coef=None, lambda_mass=1.0)
        finite += bool(np.isfinite(M).all() and np.any(M))
    assert finite > 0


@pytest.mark.gpu
@pytest.mark.parametrize("mass", [0.0, 1.0])
@pytest.mark.parametrize("hub", [0, 20])
@pytest.mark.parametrize("dim,group", [(d, g) for d in (2, 3) for g in GROUPS[d]])
def test_collapsed_elements_match_the_sequential_loop(dim, group, hub, mass):
    xyz, conn = collapsed(dim, group, hub)
    coef = np.exp(np.random.default_rng(3).standard_normal(conn.shape[0]))
    rp, ci, v = sequential(xyz, conn, coef, mass)
    assert (np.diff(rp).max() > 32) == (hub > 0)
    with femgpu.Solver() as s:
        s.set_mesh(xyz, conn)
        for _ in range(2):
            s.assemble(coef, mass)
            grp, gci, gv = s.matrix()
            assert np.array_equal(grp, rp) and np.array_equal(gci, ci)
            assert np.array_equal(gv, v, equal_nan=True)
        # a mesh of distinct vertices on the same handle
        xyz, conn = meshes.kuhn_cube(2)
        s.set_mesh(xyz, conn)
        s.assemble(None, mass)
        v = sequential(xyz, conn, None, mass)[2]
        assert np.array_equal(s.matrix()[2], v)
        assert np.array_equal(O.assemble(xyz, conn, *O.build_pattern(xyz.shape[0], conn), coef=None,
                                         lambda_mass=mass), v)
