"""Assembly and load vector against the CPU oracle, bit for bit, where their kernels change
path: last blocks of every remainder, with and without the mass term, rows past the slot
map's limit (a fan of triangles around one vertex), and coordinates so small that the
constant divisions leave their fast range.  Needs a GB300."""
import numpy as np
import pytest

import femgpu
import oracle as O
from femgpu import meshes

pytestmark = pytest.mark.gpu


def fan(k):
    """k triangles around vertex 0 (its row has k + 1 entries)."""
    t = 2 * np.pi * np.arange(k) / k
    xyz = np.zeros((k + 1, 3))
    xyz[1:, 0], xyz[1:, 1] = np.cos(t), np.sin(t)
    i = np.arange(k)
    return xyz, np.stack([0 * i, 1 + i, 1 + (i + 1) % k], axis=1).astype(np.int32)


MESHES = {
    "tet 1": lambda: meshes.kuhn_cube(1),
    "tet 4": lambda: meshes.kuhn_cube(4),  # 125 vertices: one block, three short of full
    "tet 7": lambda: meshes.kuhn_cube(7),
    "tri 10": lambda: meshes.jittered_square(10),
    "tri 23": lambda: meshes.jittered_square(23),
    "fan 31": lambda: fan(31),  # 32 entries: the longest row of the slot map
    "fan 45": lambda: fan(45),
    "tet tiny": lambda: (meshes.kuhn_cube(3)[0] * 1e-99, meshes.kuhn_cube(3)[1]),
}


@pytest.mark.parametrize("mass", [0.0, 1.0, 0.37])
@pytest.mark.parametrize("name", list(MESHES))
def test_assembly_and_load_match_oracle(name, mass):
    xyz, conn = MESHES[name]()
    rng = np.random.default_rng(3)
    coef = np.exp(rng.standard_normal(conn.shape[0]))
    f = rng.uniform(-1.0, 1.0, xyz.shape[0])
    rp, ci = O.build_pattern(xyz.shape[0], conn)
    with femgpu.Solver() as s:
        s.set_mesh(xyz, conn)
        s.assemble(coef, mass)
        grp, gci, gv = s.matrix()
        b = s.load_vector(f)
    assert np.array_equal(grp, rp) and np.array_equal(gci, ci)
    assert np.array_equal(gv, O.assemble(xyz, conn, rp, ci, coef=coef, lambda_mass=mass))
    assert np.array_equal(b, O.load_vector(xyz, conn, f))


@pytest.mark.parametrize("mesh", [("square", 89), ("square", 90), ("square", 127), ("square", 128), ("square", 180),
                                  ("fan", 341), ("fan", 342), ("fan", 2730), ("fan", 2731)])
def test_pattern_at_scan_and_sort_limits(mesh):
    # vertex counts around one and two scan tiles (8100, 8281, 16384, 16641) and beyond;
    # candidate lists around the warp's and the block's sort capacity (1024 and 8192 / 3)
    xyz, conn = meshes.jittered_square(mesh[1]) if mesh[0] == "square" else fan(mesh[1])
    rp, ci = O.build_pattern(xyz.shape[0], conn)
    with femgpu.Solver() as s:
        s.set_mesh(xyz, conn)
        s.assemble(None, 1.0)
        grp, gci, _ = s.matrix()
    assert np.array_equal(grp, rp) and np.array_equal(gci, ci)
