"""The solves that users of this package run, as cases that can be timed and checked.

Four callers reach the solve path: the 2-D pressure correction, the 3-D
projection (pressure Poisson) solve, the 1-D network solver and the adjoint of a
Darcy solve; the 3-D Stokes chain adds a saddle-point tier. Each case is one
call of such a caller with fresh inputs, on the handles (matrix, hierarchy,
batch) that its program keeps between calls. ``exact`` solves the same systems
in 64 bits with dense factorizations or a plain conjugate-gradient iteration.
"""
import functools
import math

import numpy as np
import torch

import cfdrs_b200 as cf
from cfdrs_b200 import adjoint, batch, problems

DEVICE = "cuda:0"
# A hierarchy of more rows than this is set up once per process and shared by
# the states of a case: a time-stepping program sets it up once and then solves
# for one right-hand side after the other.
SHARED_ROWS = 1_000_000


def listed():
    return [
        # The 2-D SIMPLE pressure correction with its defaults (GMRES(30), AMG
        # below 10 000 rows, host arrays): a coarse grid, where each call is
        # latency, and one just under the AMG size limit. Odd row lengths.
        {"name": "pressure_47x35", "kind": "pressure", "nx": 47, "ny": 35},
        {"name": "pressure_101x98", "kind": "pressure", "nx": 101, "ny": 98},
        # 2-D pressure Poisson by Jacobi-CG in FP64: the 128 x 128 grid of the
        # package's smallest benchmark, and a larger ragged one.
        {"name": "jacobi_cg_128x128", "kind": "jacobi_cg", "nx": 128, "ny": 128},
        {"name": "jacobi_cg_411x300", "kind": "jacobi_cg", "nx": 411, "ny": 300},
        # 3-D variable-coefficient pressure Poisson by AMG-CG: a small odd grid
        # and a large one in the mixed-precision form that production runs use,
        # a middle one in the plain FP64 form that is the drop-in default.
        {"name": "amg_cg_65_mixed", "kind": "amg_cg", "n": 65, "mixed": True},
        {"name": "amg_cg_96_fp64", "kind": "amg_cg", "n": 96, "mixed": False},
        {"name": "amg_cg_192_mixed", "kind": "amg_cg", "n": 192, "mixed": True},
        # One step of a permeability inversion: assembly from theta, hierarchy
        # refreshed for the new values, forward solve, loss, adjoint, gradient.
        {"name": "darcy_adjoint_512", "kind": "darcy", "n": 512},
        # One Picard pass over many pipe networks of uneven size: values from
        # the conductances, then every system solved; by Jacobi-CG, and by the
        # 1-D solver's own cascade (direct for small, Krylov with fallback).
        {"name": "networks_cg_768", "kind": "networks_cg", "count": 768, "nodes": 2000},
        {"name": "networks_cascade_512", "kind": "networks_cascade", "count": 512, "nodes": 2000},
        # 3-D Stokes on a staggered grid by GMRES with component blocks, the
        # first iterative tier of the saddle-point chain.
        {"name": "stokes_11", "kind": "stokes", "n": 11},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pressure", "jacobi_cg", "amg_cg", "amg_cg", "darcy", "networks_cg", "networks_cascade", "stokes"])
    if kind == "pressure":
        return {"kind": kind, "nx": rng.randint(24, 101), "ny": rng.randint(24, 98)}
    if kind == "jacobi_cg":
        return {"kind": kind, "nx": _log_int(rng, 40, 411), "ny": _log_int(rng, 40, 300)}
    if kind == "amg_cg":
        return {"kind": kind, "n": _log_int(rng, 40, 160), "mixed": rng.random() < 0.6}
    if kind == "darcy":
        return {"kind": kind, "n": _log_int(rng, 64, 512)}
    if kind == "stokes":
        return {"kind": kind, "n": rng.randint(6, 11)}
    return {"kind": kind, "count": _log_int(rng, 48, 512), "nodes": _log_int(rng, 300, 2000)}


# ---- the systems ---------------------------------------------------------------

def _field_3d(n, seed):
    """k = exp(g), g a Gaussian random field (correlation 8 cells, sigma 1)."""
    return np.exp(problems.gaussian_random_field((n, n, n), 8.0, 1.0, seed))


def _rhs(rows, seed):
    return np.random.default_rng(seed).uniform(-1.0, 1.0, rows)


@functools.lru_cache(maxsize=1)
def _shared_3d(n):
    A, _ = problems.poisson_3d_fv(n, _field_3d(n, 1))
    return A, cf.AlgebraicMultigrid(A, cf.AMGConfig.pressure_poisson())


def _poisson_3d(n, seed):
    if n ** 3 > SHARED_ROWS:
        return _shared_3d(n)
    A, _ = problems.poisson_3d_fv(n, _field_3d(n, seed))
    return A, cf.AlgebraicMultigrid(A, cf.AMGConfig.pressure_poisson())


def _theta(n, seed):
    return problems.gaussian_random_field((n, n), 16.0, 0.5, seed)


def _networks(case, seed):
    """Node counts uniform in [20, nodes], the same for every seed; trees, loop
    edges and conductances from the seed."""
    sizes = np.random.default_rng(case["count"]).integers(20, case["nodes"] + 1, case["count"])
    rng = np.random.default_rng(seed)
    return [problems.random_network_edges(int(n), rng) for n in sizes]


# ---- one case --------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "pressure":
        A, b = problems.poisson_2d_dirichlet(case["nx"], case["ny"], seed)
        disp = cf.PressureCorrectionDispatch()
        # the first call of a run sets up the hierarchy that the dispatch keeps
        disp.dispatch_solve(A, np.ones_like(b), np.zeros_like(b))
        return {"kind": kind, "A": A, "b": b, "dispatch": disp}
    if kind == "jacobi_cg":
        A, b = problems.poisson_2d_dirichlet(case["nx"], case["ny"], seed)
        pre = cf.JacobiPreconditioner(A)
        cfg = cf.IterativeSolverConfig(0.0, 1e-10, 20000)
        return {"kind": kind, "A": A, "b": torch.as_tensor(b, device=DEVICE), "pre": pre, "config": cfg}
    if kind == "amg_cg":
        A, amg = _poisson_3d(case["n"], seed)
        b = torch.as_tensor(_rhs(A.nrows, seed), device=DEVICE)
        precision = cf.Precision.FP32_REFINE if case["mixed"] else cf.Precision.FP64
        cfg = cf.IterativeSolverConfig(0.0, 1e-10, 200)
        return {"kind": kind, "A": A, "b": b, "pre": amg, "config": cfg, "precision": precision}
    if kind == "darcy":
        n = case["n"]
        pattern, _ = adjoint.darcy_2d_pattern(n)
        solver = adjoint.SparseSolver(pattern)
        theta = torch.as_tensor(_theta(n, seed), device=DEVICE).requires_grad_(True)
        # the start of an inversion: the hierarchy of the initial, uniform medium
        values, _ = adjoint.darcy_2d_assemble_device(torch.zeros_like(theta), solver)
        solver.set_values(values)
        return {"kind": kind, "n": n, "theta": theta, "solver": solver, "column": adjoint.loss_column_index(n)}
    if kind in ("networks_cg", "networks_cascade"):
        nets = batch.NetworkBatch.from_networks(_networks(case, seed))
        g = torch.as_tensor(nets.packed.conductance, device=DEVICE)
        x0 = torch.zeros(nets.rows, dtype=torch.float64, device=DEVICE)
        return {"kind": kind, "nets": nets, "g": g, "x0": x0}
    A, b, nv = problems.stokes_3d_mac(case["n"], seed=seed)
    pre = cf.ComponentBlockPreconditioner(A, nv)
    cfg = cf.IterativeSolverConfig(0.0, 1e-10, 500)
    return {"kind": kind, "A": A, "b": torch.as_tensor(b, device=DEVICE), "pre": pre, "config": cfg}


def run(state):
    kind = state["kind"]
    if kind == "pressure":
        x = np.zeros_like(state["b"])
        state["dispatch"].dispatch_solve(state["A"], state["b"], x)
        return x
    if kind == "jacobi_cg":
        x = torch.zeros_like(state["b"])
        cf.cg_preconditioned(state["A"], state["b"], state["pre"], x, state["config"])
        return x
    if kind == "amg_cg":
        x = torch.zeros_like(state["b"])
        cf.cg_preconditioned(state["A"], state["b"], state["pre"], x, state["config"], precision=state["precision"])
        return x
    if kind == "darcy":
        p = adjoint.darcy_2d_solve(state["theta"], state["solver"])
        loss = adjoint.column_loss(p, state["n"], state["column"])
        (grad,) = torch.autograd.grad(loss, state["theta"])
        return {"pressure": p.detach(), "gradient": grad}
    if kind in ("networks_cg", "networks_cascade"):
        nets, x = state["nets"], state["x0"].clone()
        nets.assemble(state["g"])
        if kind == "networks_cg":
            x, _ = nets.solve(None, x)
        else:
            x, _ = nets.solve_linear_systems(None, x, tolerance=1e-10)
        return x
    x = torch.zeros_like(state["b"])
    cf.gmres_preconditioned(state["A"], state["b"], state["pre"], x, state["config"])
    return x


def work(case):
    """The system read once, the right-hand side (or parameters) read once and
    the result written once; two operations per stored entry."""
    kind = case["kind"]
    if kind in ("pressure", "jacobi_cg"):
        rows = case["nx"] * case["ny"]
        nnz = 5 * rows
    elif kind == "amg_cg":
        rows = case["n"] ** 3
        nnz = 7 * rows
    elif kind == "darcy":
        rows = case["n"] ** 2  # theta in, pressure and gradient out
        return {"bytes": 24.0 * rows, "flops": 40.0 * rows}
    elif kind == "stokes":
        n = case["n"]
        rows = 3 * (n - 1) * n * n + n ** 3
        nnz = 3 * (n - 1) * n * n * 9 + 7 * n ** 3
    else:
        rows = case["count"] * (20 + case["nodes"]) // 2
        nnz = 3.2 * rows
        return {"bytes": 8.0 * 1.1 * rows + 8.0 * rows, "flops": 2.0 * nnz}
    return {"bytes": 12.0 * nnz + 4.0 * rows + 16.0 * rows, "flops": 2.0 * nnz}


# ---- 64-bit results --------------------------------------------------------------

def _dense(A):
    rows = np.repeat(np.arange(A.nrows), np.diff(A.row_ptr))
    D = torch.zeros((A.nrows, A.ncols), dtype=torch.float64, device=DEVICE)
    D[torch.as_tensor(rows, device=DEVICE), torch.as_tensor(A.col.astype(np.int64), device=DEVICE)] = torch.as_tensor(
        np.array(A.val), device=DEVICE)
    return D


def _dense_solve(A, b):
    D, r = _dense(A), torch.as_tensor(b, device=DEVICE)
    lu, piv = torch.linalg.lu_factor(D)
    x = torch.zeros_like(r)
    for _ in range(3):
        x = x + torch.linalg.lu_solve(lu, piv, (r - D @ x)[:, None])[:, 0]
    return x


def _cg64(A, b):
    """Jacobi-CG on a symmetric positive definite CSR matrix, restarted on the
    true residual until it no longer falls."""
    S = torch.sparse_csr_tensor(torch.as_tensor(A.row_ptr, device=DEVICE),
                                torch.as_tensor(A.col.astype(np.int64), device=DEVICE),
                                torch.as_tensor(np.array(A.val), device=DEVICE), size=A.shape)
    d = 1.0 / torch.as_tensor(A.diagonal(), device=DEVICE)
    x = torch.zeros_like(b)
    for _ in range(3):
        r = b - S @ x
        z = d * r
        p, rho, r0 = z.clone(), torch.dot(r, z), torch.linalg.vector_norm(r)
        e = torch.zeros_like(x)
        for it in range(20000):
            q = S @ p
            alpha = rho / torch.dot(p, q)
            e += alpha * p
            r -= alpha * q
            if it % 50 == 49 and float(torch.linalg.vector_norm(r)) <= 1e-9 * float(r0):
                break
            z = d * r
            new = torch.dot(r, z)
            p = z + (new / rho) * p
            rho = new
        x = x + e
    return x


def _darcy_apply(theta, p):
    """A(theta) p - b(theta) of the finite-volume Darcy system, cell by cell."""
    k = torch.exp(theta)
    fx = 2.0 * k[:, :-1] * k[:, 1:] / (k[:, :-1] + k[:, 1:])
    fy = 2.0 * k[:-1] * k[1:] / (k[:-1] + k[1:])
    qx, qy = fx * (p[:, :-1] - p[:, 1:]), fy * (p[:-1] - p[1:])
    pad = torch.nn.functional.pad
    out = pad(qx, (0, 1)) - pad(qx, (1, 0)) + pad(qy, (0, 0, 0, 1)) - pad(qy, (0, 0, 1, 0))
    n = theta.shape[0]
    left, right = 2.0 * k[:, :1] * (p[:, :1] - 1.0), 2.0 * k[:, -1:] * p[:, -1:]
    return out + pad(left, (0, n - 1)) + pad(right, (n - 1, 0))


def exact(case, seed):
    kind = case["kind"]
    if kind == "pressure":
        A, b = problems.poisson_2d_dirichlet(case["nx"], case["ny"], seed)
        return _dense_solve(A, b).cpu().numpy()
    if kind == "jacobi_cg":
        A, b = problems.poisson_2d_dirichlet(case["nx"], case["ny"], seed)
        return _cg64(A, torch.as_tensor(b, device=DEVICE))
    if kind == "amg_cg":
        n = case["n"]
        A, _ = problems.poisson_3d_fv(n, _field_3d(n, 1 if n ** 3 > SHARED_ROWS else seed))
        return _cg64(A, torch.as_tensor(_rhs(A.nrows, seed), device=DEVICE))
    if kind == "darcy":
        n, th = case["n"], _theta(case["n"], seed)
        A, b = problems.darcy_2d(th)
        p = _cg64(A, torch.as_tensor(b, device=DEVICE))
        g = torch.zeros((n, n), dtype=torch.float64, device=DEVICE)
        c = math.ceil(0.75 * n - 0.5)
        g[:, c] = 2.0 * p.reshape(n, n)[:, c]
        lam = _cg64(A, g.reshape(-1)).reshape(n, n)
        theta = torch.as_tensor(th, device=DEVICE).requires_grad_(True)
        (grad,) = torch.autograd.grad((lam * _darcy_apply(theta, p.reshape(n, n))).sum(), theta)
        return {"pressure": p, "gradient": -grad}
    if kind in ("networks_cg", "networks_cascade"):
        out = []
        for net in _networks(case, seed):
            A, b = net.assemble()
            out.append(_dense_solve(A, b))
        return torch.cat(out)
    A, b, _ = problems.stokes_3d_mac(case["n"], seed=seed)
    return _dense_solve(A, b)
