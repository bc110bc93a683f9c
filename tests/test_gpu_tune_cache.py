"""A tuning file (FEMGPU_TUNE_CACHE) whose values are not lane counts changes no result: they are
measured again.  Each file is read by a process of its own.  Needs a GB300."""
import os
import re
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = """
import hashlib, sys
sys.path.insert(0, "sci-solver_fem_gb300")
import numpy as np, femgpu
from femgpu import meshes
for precision in (0, 1):
    xyz, conn, kappa, f, mask = meshes.poisson3d_problem(17, sigma=1.0)
    s = femgpu.Solver(solverType=1, seed=1, precision=precision)
    s.set_mesh(xyz, conn)
    s.assemble(kappa, 0.0)
    s.set_dirichlet(mask)
    s.setup()
    z = s.vcycle(np.random.default_rng(1).standard_normal(xyz.shape[0]))
    print("z", hashlib.sha256(z.tobytes()).hexdigest())
"""


def run(path):
    env = dict(os.environ, FEMGPU_TUNE_CACHE=str(path))
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=300, cwd=ROOT, env=env)
    assert r.returncode == 0, r.stderr
    return re.findall(r"^z (\w+)$", r.stdout, re.M)


def test_values_that_are_no_lane_counts(tmp_path):
    good = tmp_path / "good"
    z = run(good)
    lines = good.read_text().splitlines()
    assert len(z) == 2 and len(lines) >= 2 and all("|lanes|" in l for l in lines)
    assert run(good) == z and good.read_text().splitlines() == lines  # read back, nothing measured again
    for value in ("3", "0", "-4", "48", "64", "4", "32"):
        path = tmp_path / f"v{value}"
        path.write_text("".join(f"{l.rsplit(' ', 1)[0]} {value}\n" for l in lines))
        assert run(path) == z, value
