"""The calls whose time this framework is judged by, with their inputs and what they compute.

Kinds of case (`kind`):
  solve     AMG setup and PCG solve of an assembled operator, right-hand side and solution in
            device memory: the loop of a program whose coefficients change from solve to solve
  remesh    the whole host flow of the reference's FEMSolver on a new mesh: pattern, assembly of
            K + M, load vector, setup, solve; host arrays in and out
  multi     many right-hand sides with a hierarchy that the program keeps
  grad      forward solve and adjoint gradient through the PyTorch binding
  assemble  new coefficients on a kept mesh: assembly, then y = A u (a nonlinear residual)
  step      a time step with the reference's default solver (one V-cycle): load vector, A u,
            V-cycle of the load

Meshes are unit squares of jittered triangles (dim 2) and Kuhn-split unit cubes (dim 3) with `n`
cells per edge.  `shuffled` numbers the vertices at random, as a mesh file of an unstructured
mesher may, and moves interior vertices by up to 0.1 h.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sci-solver_fem_gb300"))

import femgpu  # noqa: E402
from femgpu import meshes  # noqa: E402
from femgpu.autograd import fem_solve  # noqa: E402

TOL = 1e-8
LABEL_COEF = (1.0, 1.0, 2.0, 3.0, 4.0, 5.0, 6.0)  # material label -> coefficient


def listed():
    return [
        # the plain 2D Poisson problem: small, so launches and round trips count
        dict(name="solve_2d_64_fp64", kind="solve", dim=2, n=64, precision=1, smoother=0, sigma=0.0, shuffled=False),
        # the smallest 3D problems, a few thousand unknowns
        dict(name="solve_3d_13", kind="solve", dim=3, n=13, precision=0, smoother=0, sigma=1.0, shuffled=False),
        # an ordinary plane problem with the point smoother
        dict(name="solve_2d_300_l1", kind="solve", dim=2, n=300, precision=0, smoother=1, sigma=1.0, shuffled=False),
        # an ordinary size on an irregular mesh with the point smoother
        dict(name="solve_3d_50_l1", kind="solve", dim=3, n=50, precision=0, smoother=1, sigma=1.0, shuffled=True),
        # plain FP64 at the middle size
        dict(name="solve_3d_64_fp64", kind="solve", dim=3, n=64, precision=1, smoother=0, sigma=1.0, shuffled=False),
        # the headline problem: 2.1 M unknowns, coefficients over five decades
        dict(name="solve_3d_128", kind="solve", dim=3, n=128, precision=0, smoother=0, sigma=2.0, shuffled=False),
        # a new mesh from the host, solved once
        dict(name="remesh_3d_33", kind="remesh", dim=3, n=33, shuffled=True),
        # 64 load cases on one operator
        dict(name="multi_3d_64", kind="multi", dim=3, n=64, precision=0, rhs=64, sigma=1.0),
        # inverse problem: forward solve and gradient with respect to 5.3 M log-coefficients
        dict(name="grad_3d_96", kind="grad", dim=3, n=96, sigma=1.0),
        # new coefficients, then the operator's action
        dict(name="assemble_3d_101", kind="assemble", dim=3, n=101, mass=1.0, shuffled=False),
        dict(name="assemble_2d_500", kind="assemble", dim=2, n=500, mass=1.0, shuffled=False),
        # a time step by one V-cycle
        dict(name="step_3d_60", kind="step", dim=3, n=60, precision=0, shuffled=False),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "remesh", "multi", "grad", "assemble", "step"])
    if kind == "solve":
        dim = rng.choice([2, 3, 3])
        fp64 = rng.random() < 0.3
        n = _size(rng, 16, 400) if dim == 2 else _size(rng, 8, 80 if fp64 else 127)
        point = dim == 2 or rng.random() < 0.25
        return dict(kind=kind, dim=dim, n=n, precision=int(fp64), smoother=int(point),
                    sigma=round(rng.uniform(0.0, 1.0 if dim == 2 else 2.0), 2),
                    shuffled=n <= 80 and rng.random() < 0.4)
    if kind == "remesh":
        dim = rng.choice([2, 3, 3])
        return dict(kind=kind, dim=dim, n=_size(rng, 16, 300) if dim == 2 else _size(rng, 8, 60),
                    shuffled=rng.random() < 0.5)
    if kind == "multi":
        return dict(kind=kind, dim=3, n=_size(rng, 10, 60), precision=int(rng.random() < 0.3), rhs=rng.randint(2, 64),
                    sigma=round(rng.uniform(0.0, 2.0), 2))
    if kind == "grad":
        dim = rng.choice([2, 3, 3])
        return dict(kind=kind, dim=dim, n=_size(rng, 16, 300) if dim == 2 else _size(rng, 8, 95),
                    sigma=round(rng.uniform(0.2, 1.2), 2))
    if kind == "assemble":
        dim = rng.choice([2, 3, 3])
        n = _size(rng, 32, 900) if dim == 2 else _size(rng, 10, 127)
        return dict(kind=kind, dim=dim, n=n, mass=rng.choice([0.0, 1.0]), shuffled=n <= 80 and rng.random() < 0.4)
    return dict(kind=kind, dim=3, n=_size(rng, 8, 70), precision=int(rng.random() < 0.3), shuffled=rng.random() < 0.4)


# ---- inputs ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=64)
def _mesh(dim, n, shuffled):
    """Coordinates, elements and Dirichlet mask (2D: the boundary, 3D: z = 0)."""
    if dim == 2:
        xyz, conn = meshes.jittered_square(n)
        mask = meshes.boundary_mask_2d(n)
    else:
        xyz, conn = meshes.kuhn_cube(n)
        mask = meshes.bottom_face_mask(n)
    if shuffled:
        r = np.random.default_rng(n)
        if dim == 3:
            inner = ((xyz > 0.0) & (xyz < 1.0)).all(axis=1)
            xyz = xyz.copy()
            xyz[inner] += r.uniform(-0.1 / n, 0.1 / n, size=(int(inner.sum()), 3))
        new = r.permutation(xyz.shape[0]).astype(np.int32)
        moved, m = np.empty_like(xyz), np.empty_like(mask)
        moved[new], m[new] = xyz, mask
        xyz, mask, conn = moved, m, new[conn]
    return xyz, conn, mask


def _gen(seed, which=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * (int(seed) + 1) + which)


def _normal(count, seed, which):
    return torch.randn(count, dtype=torch.float64, device="cuda", generator=_gen(seed, which))


def _uniform(shape, seed, which):
    return torch.rand(shape, dtype=torch.float64, device="cuda", generator=_gen(seed, which)) * 2.0 - 1.0


def _load(s, f, mask):
    b = s.load_vector(f.cpu().numpy())
    b[mask.astype(bool)] = 0.0
    return b


def _smoother(point):
    """The point (l1-Jacobi) smoother with two sweeps, or the default partition smoother with five."""
    return dict(smoother=1, preInnerIters=2, postInnerIters=2) if point else {}


def _assembled(xyz, conn, mask, coef, **options):
    s = femgpu.Solver(solverType=1, tolerance=TOL, maxIters=1000, flexibleCG=1, seed=1, **options)
    s.set_mesh(xyz, conn)
    torch.cuda.synchronize()
    s.assemble_device(coef.data_ptr(), 0.0)
    s.set_dirichlet(mask)
    return s


def prepare(case, seed):
    c = dict(case)
    st = dict(case=c)
    xyz, conn, mask = _mesh(c["dim"], c["n"], c.get("shuffled", False))
    nv, ne = xyz.shape[0], conn.shape[0]
    st["stream"] = torch.cuda.Stream()
    own = dict(stream=st["stream"].cuda_stream)
    if c["kind"] == "solve":
        coef = torch.exp(c["sigma"] * _normal(ne, seed, 0))
        s = _assembled(xyz, conn, mask, coef, precision=c["precision"], **_smoother(c["smoother"]), **own)
        st["b"] = torch.from_numpy(_load(s, _uniform(nv, seed, 1), mask)).cuda()
        st["x"] = torch.zeros_like(st["b"])
    elif c["kind"] == "remesh":
        s = femgpu.Solver(solverType=1, tolerance=TOL, maxIters=1000, flexibleCG=1, seed=1, **_smoother(c["dim"] == 2))
        st["mesh"] = (xyz, conn)
        st["labels"] = np.random.default_rng(seed).integers(0, 7, size=ne).astype(np.int32)
        st["f"] = _uniform(nv, seed, 1).cpu().numpy()
    elif c["kind"] == "multi":
        coef = torch.exp(c["sigma"] * _normal(ne, seed, 0))
        s = _assembled(xyz, conn, mask, coef, precision=c["precision"], **own)
        s.setup()
        st["b"] = _uniform((c["rhs"], nv), seed, 1) / nv
        st["b"][:, torch.from_numpy(mask.astype(bool)).cuda()] = 0.0
        st["x"] = torch.zeros_like(st["b"])
    elif c["kind"] == "grad":
        s = femgpu.Solver(solverType=1, tolerance=1e-10, maxIters=1000, flexibleCG=1, seed=1,
                          **_smoother(c["dim"] == 2))
        s.set_mesh(xyz, conn)
        st["theta"] = (c["sigma"] * _normal(ne, seed, 0)).requires_grad_(True)
        st["b"] = torch.from_numpy(_load(s, _uniform(nv, seed, 1), mask)).cuda()
        st["mask"] = mask
        st["at"] = _observed(nv)
        st["obs"] = 1e-3 * _normal(st["at"].numel(), seed, 2)
    else:
        s = femgpu.Solver(solverType=0, flexibleCG=1, seed=1, precision=c.get("precision", 0), **own)
        s.set_mesh(xyz, conn)
        st["coef"] = torch.exp(_normal(ne, seed, 0))
        st["u"] = _uniform(nv, seed, 1)
        st["y"] = torch.empty_like(st["u"])
        if c["kind"] == "step":
            torch.cuda.synchronize()
            s.assemble_device(st["coef"].data_ptr(), 1.0)
            s.setup()
            st["f"] = _uniform(nv, seed, 2)
            st["b"] = torch.empty_like(st["u"])
            st["x"] = torch.empty_like(st["u"])
    st["solver"] = s
    torch.cuda.synchronize()
    return st


def _observed(nv):
    pick = np.random.default_rng(10).choice(nv, max(1, nv // 100), replace=False)
    return torch.from_numpy(np.sort(pick)).cuda()


def run(state):
    c = state["case"]
    kind = c["kind"]
    s = state["solver"]
    if kind == "remesh":
        s.set_mesh(*state["mesh"], labels=state["labels"])
        s.assemble()
        b = s.load_vector(state["f"])
        s.setup()
        x, _ = s.solve(b)
        return {"b": b, "x": x}
    if kind == "grad":
        theta = state["theta"]
        u = fem_solve(s, theta, state["b"], state["mask"])
        loss = 0.5 * (u[state["at"]] - state["obs"]).square().sum()
        (g,) = torch.autograd.grad(loss, theta)
        return {"u": u.detach(), "grad": g}
    with torch.cuda.stream(state["stream"]):
        if kind == "solve":
            s.setup()
            state["x"].zero_()
            s.solve_device(state["b"].data_ptr(), state["x"].data_ptr())
            return state["x"]
        if kind == "multi":
            b, x = state["b"], state["x"]
            x.zero_()
            s.solve_multi_device(b.shape[0], b.data_ptr(), b.shape[1], x.data_ptr(), x.shape[1])
            return x
        if kind == "assemble":
            s.assemble_device(state["coef"].data_ptr(), c["mass"])
            s.spmv_device(state["u"].data_ptr(), state["y"].data_ptr())
            return state["y"]
        s.load_vector_device_noalloc(state["f"].data_ptr(), state["b"].data_ptr())
        s.spmv_device(state["u"].data_ptr(), state["y"].data_ptr())
        s.solve_device(state["b"].data_ptr(), state["x"].data_ptr())
        return {"b": state["b"], "y": state["y"], "x": state["x"]}


# ---- what a pass cannot do without ---------------------------------------------------
def _counts(dim, n):
    """Vertices, elements and operator entries (with the diagonal) of a mesh of n cells per edge."""
    m = n + 1
    if dim == 2:  # edges: 2 n m along the axes, n^2 diagonals
        return m * m, 2 * n * n, m * m + 2 * (2 * n * m + n * n)
    # edges: 3 n m^2 along the axes, 3 n^2 m face diagonals, n^3 body diagonals
    return m ** 3, 6 * n ** 3, m ** 3 + 2 * (3 * n * m * m + 3 * n * n * m + n ** 3)


def work(case):
    """Inputs read once and outputs written once; the flops of one product with the operator
    per solved column (iterations are the method's, not the problem's)."""
    c = case
    v, e, z = _counts(c["dim"], c["n"])
    k = c["dim"] + 1
    mesh = 24 * v + 4 * k * e
    element = 200 if c["dim"] == 3 else 120
    if c["kind"] == "solve":
        return {"bytes": 12.0 * z + 20 * v, "flops": 2.0 * z}
    if c["kind"] == "remesh":
        return {"bytes": float(mesh + 4 * e + 24 * v), "flops": float(element * e + 2 * z)}
    if c["kind"] == "multi":
        return {"bytes": 12.0 * z + 4 * v + 16.0 * v * c["rhs"], "flops": 2.0 * z * c["rhs"]}
    if c["kind"] == "grad":
        return {"bytes": float(mesh + 16 * e + 17 * v), "flops": float(2 * element * e + 4 * z)}
    if c["kind"] == "assemble":  # mesh and coefficients in, the operator's values and y out
        return {"bytes": float(mesh + 8 * e + 8 * z + 16 * v), "flops": float(element * e + 2 * z)}
    return {"bytes": float(mesh + 12 * z + 4 * v + 40 * v), "flops": float(30 * e + 4 * z)}


# ---- the same in 64 bits, without the framework's code -----------------------------------
def _gradients(xyz, conn):
    """P1 basis gradients (ne, k, d) and element measures."""
    d = conn.shape[1] - 1
    p = xyz[conn.long()][:, :, :d]
    edges = p[:, 1:] - p[:, :1]
    g = torch.linalg.inv(edges).transpose(1, 2)
    g = torch.cat([-g.sum(dim=1, keepdim=True), g], dim=1)
    return g, torch.linalg.det(edges).abs() / math.factorial(d)


def _operator(xyz, conn, coef, mass):
    """sum_e c_e K_e + mass M_e as a sparse CSR matrix."""
    g, vol = _gradients(xyz, conn)
    k = conn.shape[1]
    nv = xyz.shape[0]
    el = (coef * vol)[:, None, None] * (g @ g.transpose(1, 2))
    del g
    if mass:
        m = (torch.ones(k, k, device="cuda", dtype=torch.float64) + torch.eye(k, device="cuda", dtype=torch.float64))
        el = el + mass * vol[:, None, None] * m / (k * (k + 1))
    ij = conn.long()
    key = (ij[:, :, None] * nv + ij[:, None, :]).reshape(-1)
    key, at = torch.unique(key, return_inverse=True)
    val = torch.zeros(key.numel(), dtype=torch.float64, device="cuda").index_add_(0, at, el.reshape(-1))
    rows, cols = key // nv, key % nv
    return rows, cols, val


def _csr(rows, cols, val, nv):
    rp = torch.zeros(nv + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=nv), 0)
    return torch.sparse_csr_tensor(rp, cols, val, size=(nv, nv))


def _eliminated(rows, cols, val, mask):
    """Rows and columns of the masked vertices zeroed, with a unit diagonal."""
    hit = mask[rows] | mask[cols]
    return torch.where(hit, (rows == cols).to(val.dtype), val)


def _solved(rows, cols, val, b, tol=1e-13, most=20000):
    """Jacobi-preconditioned CG on the columns of b (nv, k)."""
    nv = b.shape[0]
    A = _csr(rows, cols, val, nv)
    on = rows == cols
    inv = torch.empty(nv, dtype=torch.float64, device="cuda")
    inv[rows[on]] = 1.0 / val[on]
    inv = inv[:, None]
    x = torch.zeros_like(b)
    r = b.clone()
    z = inv * r
    p = z.clone()
    rz = (r * z).sum(0)
    goal = tol * b.norm(dim=0)
    for it in range(most):
        y = A @ p
        a = rz / (p * y).sum(0).clamp_min(1e-300)
        x += a * p
        r -= a * y
        if it % 25 == 24 and bool((r.norm(dim=0) <= goal).all()):
            break
        z = inv * r
        new = (r * z).sum(0)
        p = z + (new / rz.clamp_min(1e-300)) * p
        rz = new
    return x


def _load64(xyz, conn, f):
    _, vol = _gradients(xyz, conn)
    k = conn.shape[1]
    fe = f[conn.long()]
    part = (vol / (k * (k + 1)))[:, None] * (fe.sum(1, keepdim=True) + fe)
    return torch.zeros_like(f).index_add_(0, conn.long().reshape(-1), part.reshape(-1))


def exact(case, seed):
    c = case
    xyz, conn, mask = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in _mesh(c["dim"], c["n"], c.get("shuffled", False)))
    mask = mask.bool()
    nv, ne = xyz.shape[0], conn.shape[0]
    if c["kind"] in ("solve", "multi"):
        rows, cols, val = _operator(xyz, conn, torch.exp(c["sigma"] * _normal(ne, seed, 0)), 0.0)
        if c["kind"] == "solve":
            b = _load64(xyz, conn, _uniform(nv, seed, 1))[:, None]
        else:
            b = (_uniform((c["rhs"], nv), seed, 1) / nv).T.contiguous()
        b[mask] = 0.0
        x = _solved(rows, cols, _eliminated(rows, cols, val, mask), b)
        return x[:, 0] if c["kind"] == "solve" else x.T.contiguous()
    if c["kind"] == "remesh":
        label = np.random.default_rng(seed).integers(0, 7, size=ne)
        # labels choose the coefficient of tetrahedra only
        coef = torch.tensor(LABEL_COEF, dtype=torch.float64, device="cuda")[torch.from_numpy(label).cuda()] \
            if c["dim"] == 3 else torch.ones(ne, dtype=torch.float64, device="cuda")
        rows, cols, val = _operator(xyz, conn, coef, 1.0)
        b = _load64(xyz, conn, _uniform(nv, seed, 1))
        return {"b": b, "x": _solved(rows, cols, val, b[:, None])[:, 0]}
    if c["kind"] == "grad":
        coef = torch.exp(c["sigma"] * _normal(ne, seed, 0))
        rows, cols, val = _operator(xyz, conn, coef, 0.0)
        val = _eliminated(rows, cols, val, mask)
        b = _load64(xyz, conn, _uniform(nv, seed, 1))
        b[mask] = 0.0
        u = _solved(rows, cols, val, b[:, None])[:, 0]
        at = _observed(nv)
        r = torch.zeros_like(u)
        r[at] = u[at] - 1e-3 * _normal(at.numel(), seed, 2)
        r[mask] = 0.0
        lam = _solved(rows, cols, val, r[:, None])[:, 0]
        g, vol = _gradients(xyz, conn)
        gu = (u[conn.long()][:, :, None] * g).sum(1)
        gl = (lam[conn.long()][:, :, None] * g).sum(1)
        return {"u": u, "grad": -coef * vol * (gu * gl).sum(1)}
    rows, cols, val = _operator(xyz, conn, torch.exp(_normal(ne, seed, 0)), c.get("mass", 1.0))
    y = (_csr(rows, cols, val, nv) @ _uniform(nv, seed, 1)[:, None])[:, 0]
    if c["kind"] == "assemble":
        return y
    return {"b": _load64(xyz, conn, _uniform(nv, seed, 2)), "y": y, "x": None}
