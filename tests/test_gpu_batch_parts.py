"""Batches longer than one part (six handles share a graph): results, statuses and graph times
by part, on a GB300; and the number of handles that the benchmark's batch of meshes gives to one
call, on the CPU."""
import argparse
import importlib
import json

import numpy as np
import pytest

import femgpu
from conftest import ROOT
from femgpu import meshes

PART = 6


def problem(n, seed, **opts):
    xyz, conn, kappa, f, mask = meshes.poisson3d_problem(n, sigma=1.0, kappa_seed=seed, f_seed=1000 + seed)
    s = femgpu.Solver(solverType=1, tolerance=1e-8, maxIters=300, flexibleCG=1, seed=1, **opts)
    s.set_mesh(xyz, conn)
    s.assemble(kappa, 0.0)
    s.set_dirichlet(mask)
    return s, np.where(mask.astype(bool), 0.0, s.load_vector(f))


@pytest.mark.gpu
@pytest.mark.parametrize("count", [PART, PART + 1, 2 * PART + 1])
def test_parts_match_single_solves(count):
    sizes = np.random.default_rng(11).integers(3, 7, size=count)
    probs = [problem(int(n), 50 + i) for i, n in enumerate(sizes)]
    solvers, bs = [p[0] for p in probs], [p[1] for p in probs]
    single = []
    for s, b in probs:
        s.setup()
        single.append(s.solve(b))
    # new hierarchies and graphs, the kept graphs, new hierarchies again
    for setup in (True, False, True):
        xs, stats, status = femgpu.solve_batch(solvers, bs, setup=setup)
        assert status == 0
        for x, st, (x1, st1) in zip(xs, stats, single):
            assert np.array_equal(x, x1) and st["iterations"] == st1["iterations"] and st["relres"] <= 1e-8
        times = [st["solve_ms"] for st in stats]  # the time of the graph that holds the problem
        parts = [set(times[i:i + PART]) for i in range(0, count, PART)]
        assert all(len(p) == 1 for p in parts) and len(set.union(*parts)) == len(parts)


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [0, PART])
def test_a_failing_problem_leaves_the_other_parts(bad):
    probs = [problem(4, 70 + i) for i in range(PART + 2)]
    probs[bad] = (femgpu.Solver(solverType=1), np.ones(8))  # no operator
    xs, stats, status = femgpu.solve_batch([p[0] for p in probs], [p[1] for p in probs],
                                           x0s=[np.zeros(p[1].shape[0]) for p in probs], check=False)
    assert status == 3  # FEMGPU_ERR_NOT_READY
    for i, (s, b) in enumerate(probs):
        if i != bad:
            assert np.array_equal(xs[i], s.solve(b)[0]) and stats[i]["relres"] <= 1e-8


@pytest.mark.gpu
@pytest.mark.parametrize("other", [1, PART])
def test_a_repeated_handle_in_any_part_is_refused(other):
    probs = [problem(3, 90 + i) for i in range(PART + 1)]
    probs[other] = probs[0]
    _, _, status = femgpu.solve_batch([p[0] for p in probs], [p[1] for p in probs], check=False)
    assert status == 1  # FEMGPU_ERR_INVALID, before any work


class _FakeSolver:
    def __init__(self, **options):
        pass

    def set_mesh(self, xyz, conn):
        pass

    def assemble(self, kappa, mass):
        pass

    def set_dirichlet(self, mask):
        pass

    def load_vector(self, f):
        return f


def test_bench_meshes_are_solved_in_calls_of_a_part(monkeypatch, capsys):
    monkeypatch.syspath_prepend(ROOT)
    bench = importlib.import_module("bench")
    calls = []

    def solve_batch(solvers, bs, **options):
        assert len(solvers) == len(bs)
        calls.append(len(solvers))
        stat = dict(iterations=1, relres=0.0, setup_ms=1.0, solve_ms=1.0)
        return bs, [stat] * len(solvers), 0

    monkeypatch.setattr(femgpu, "Solver", _FakeSolver)
    monkeypatch.setattr(femgpu, "solve_batch", solve_batch)
    monkeypatch.setattr(meshes, "poisson3d_problem", lambda m, **seeds: (
        np.zeros((m, 3)), np.zeros((1, 4), np.int32), np.ones(1), np.ones(m), np.zeros(m, np.uint8)))
    bench.run_meshes(argparse.Namespace(warmup=1, steps=2))
    out = json.loads(capsys.readouterr().out)
    assert max(calls) <= PART and sum(calls) == 48 * (1 + 2) * 2  # two timings of three steps
    assert out["config"]["meshes"] == 48 and out["pcg_iterations_total"] == 48
