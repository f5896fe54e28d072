"""Workloads of the sparse direct solver that its speed is measured on.

The matrices are the families of pastix_b200.gen (3D 7-point Laplacian, 2D
variable-coefficient diffusion, 27-point convection-diffusion, 3-unknown
elastic stencil), ordered by grid nested dissection.  A program that solves a
sequence of systems (time steps, Newton or optimisation steps) analyses its
pattern once and keeps the handle, so the handle of the pattern in use is kept
here too; the numerical values, right-hand sides and adjoint seeds come from
the seed alone.  New values are D A D with D a positive diagonal, which keeps
the pattern, the symmetry and the inertia.

Right-hand sides are b = A x for a drawn x, so the exact solution is known: the
rounding of b moves it by cond(A) * 1e-16.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pastix_b200 import gen
from pastix_b200 import pastix as px
from pastix_b200.autograd import SparseSolver, solve as diff_solve
from pastix_b200.spm import mtxtype, spmatrix

FACT = {"POTRF": px.factotype.POTRF, "SYTRF": px.factotype.SYTRF, "GETRF": px.factotype.GETRF}
TARGET = 1e-12  # ||b - A x|| / ||b|| at which refinement stops


def _case(name, call, matrix, nx, ny, nz, fact, nrhs, mixed):
    c = {"call": call, "matrix": matrix, "nx": nx, "ny": ny, "nz": nz, "fact": fact, "nrhs": nrhs, "mixed": mixed}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a small system solved again and again (a time step of a coarse model): launches and latency count
        _case("lap20_llt_f64", "factor_solve", "lap", 20, 20, 20, "POTRF", 1, False),
        # the same step through the C API's host buffers on a ragged grid, as a PaStiX program calls it
        _case("lap61x47x53_host", "host", "lap", 61, 47, 53, "POTRF", 1, False),
        # the headline system, n = 10^6: plain FP64 factorization and solve
        _case("lap100_llt_f64", "factor_solve", "lap", 100, 100, 100, "POTRF", 1, False),
        # the headline system by FP32 factors and FP64 CG refinement
        _case("lap100_llt_mixed", "factor_refine", "lap", 100, 100, 100, "POTRF", 1, True),
        # gradient of a PDE-constrained loss: forward solve, transposed solve, value gradient
        _case("grf512_adjoint", "adjoint", "grf", 512, 512, 1, "POTRF", 1, False),
        # unsymmetric transport problem, several right-hand sides, FP32 factors and GMRES(30)
        _case("cd64_lu_mixed", "factor_refine", "cd", 64, 64, 64, "GETRF", 4, True),
        # the same family in plain FP64 LU on a ragged grid
        _case("cd45x38x41_lu_f64", "factor_solve", "cd", 45, 38, 41, "GETRF", 4, False),
        # shifted (indefinite) structure, many load cases, LDL^T in FP64
        _case("el32_ldlt_f64", "factor_solve", "el", 32, 32, 32, "SYTRF", 64, False),
        # the same structure at a smaller size by FP32 factors and GMRES(30)
        _case("el20x23x18_ldlt_mixed", "factor_refine", "el", 20, 23, 18, "SYTRF", 1, True),
        # factors kept, new right-hand sides: a block of 16 in FP64
        _case("lap80_solve16_f64", "solve", "lap", 80, 80, 80, "POTRF", 16, False),
        # residual r = b - A x of the caller's own iteration
        _case("lap80_residual", "spmv", "lap", 80, 80, 80, "POTRF", 1, False),
        # factors kept: FP32 factors applied once, as the preconditioner of the caller's own iteration
        _case("lap100_solve_f32", "solve", "lap", 100, 100, 100, "POTRF", 1, True),
    ]


def _grid(rng, lo, hi, dims):
    """A grid of about lo .. hi vertices (logarithmic), sides within a factor of two of each other."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    w = [math.exp(rng.uniform(-0.34, 0.34)) for _ in range(dims)]
    s = (n / math.prod(w)) ** (1.0 / dims)
    side = [max(6, int(s * v)) for v in w] + [1] * (3 - dims)
    while math.prod(side) > hi:
        side[side.index(max(side))] -= 1
    return side


def draw(rng):
    kind = rng.choice(["lap_f64", "lap_mixed", "adjoint", "lu_mixed", "lu_f64", "ldlt", "solve", "host"])
    if kind == "lap_f64":
        return _case(None, "factor_solve", "lap", *_grid(rng, 8000, 500000, 3), "POTRF", rng.choice([1, 1, 16]), False)
    if kind == "lap_mixed":
        return _case(None, "factor_refine", "lap", *_grid(rng, 8000, 800000, 3), "POTRF", rng.choice([1, 1, 16]), True)
    if kind == "adjoint":
        return _case(None, "adjoint", "grf", *_grid(rng, 64 * 64, 512 * 512, 2), "POTRF", 1, False)
    if kind == "lu_mixed":
        return _case(None, "factor_refine", "cd", *_grid(rng, 4000, 64 ** 3, 3), "GETRF", rng.choice([1, 4]), True)
    if kind == "lu_f64":
        return _case(None, "factor_solve", "cd", *_grid(rng, 4000, 100000, 3), "GETRF", rng.choice([1, 4]), False)
    if kind == "ldlt":
        return _case(None, "factor_solve", "el", *_grid(rng, 1000, 32 ** 3, 3), "SYTRF", rng.choice([1, 7, 64]), False)
    if kind == "solve":
        return _case(None, "solve", "lap", *_grid(rng, 8000, 500000, 3), "POTRF", rng.randint(1, 16),
                     rng.random() < 0.5)
    return _case(None, "host", "lap", *_grid(rng, 8000, 250000, 3), "POTRF", rng.choice([1, 3]), False)


# ---- the pattern in use ----
def _matrix(case):
    m, g = case["matrix"], (case["nx"], case["ny"], case["nz"])
    if m == "lap":
        return gen.laplacian7(*g)
    if m == "grf":
        return gen.diffusion5_grf(g[0], g[1], np.exp(gen.grf_2d(g[0], g[1], 16.0, 1.0, 2)))
    if m == "cd":
        return gen.convdiff27(*g)
    return gen.elastic27_dof3(*g)[0]


class _Handle:
    """The analysed pattern of one workload, as a program that solves many systems keeps it."""

    def __init__(self, case):
        self.A, self.lu = _matrix(case), case["fact"] == "GETRF"
        grid = (case["nx"], case["ny"], case["nz"])
        if case["call"] == "adjoint":
            self.solver = SparseSolver(self.A, case["fact"], grid=grid)
            self.pd = self.solver.pd
        else:
            ip, dp = px.initParam()
            ip[px.iparm.factorization] = FACT[case["fact"]]
            ip[px.iparm.mixed] = int(case["mixed"])
            ip[px.iparm.refinement] = px.refine.CG if case["fact"] == "POTRF" else px.refine.GMRES
            ip[px.iparm.gmres_im] = 30
            dp[px.dparm.epsilon_refinement] = TARGET
            self.pd = px.init(ip, dp)
            px.analyze_grid(self.pd, self.spm(np.ones(self.A.shape[0]))[0], *grid)
        self.factored = False

    def spm(self, d):
        """The matrix D A D as the library takes it, and whole."""
        A = self.A.copy()
        cols = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))
        A.data = A.data * d[A.indices] * d[cols]
        return spmatrix(A, mtxtype.General if self.lu else mtxtype.Symmetric), A

    def __del__(self):
        px.finalize(self.pd)


_handles = {}


def _key(case):
    kept = {"spmv": "solve"}.get(case["call"], case["call"])  # both work on the kept factors' matrix
    return (kept,) + tuple(v for k, v in sorted(case.items()) if k not in ("name", "nrhs", "call"))


def _handle(case):
    key = _key(case)
    if key not in _handles:
        _handles.clear()  # one pattern at a time; states of an earlier one keep theirs
        _handles[key] = _Handle(case)
    return _handles[key]


def _truth(case, seed):
    """Scaling and true solutions (n x nrhs; adjoint: the solution and the adjoint state)."""
    rng = np.random.default_rng([seed, 77])
    n = case["nx"] * case["ny"] * case["nz"] * (3 if case["matrix"] == "el" else 1)
    d = rng.uniform(0.8, 1.25, n)
    x = rng.uniform(-1.0, 1.0, (2 if case["call"] == "adjoint" else case["nrhs"], n)).T  # column major
    return d, x


def _system(case, seed):
    """Handle, matrix and right-hand sides for a seed; kept factors belong to one fixed matrix."""
    h = _handle(case)
    d, x = _truth(case, seed)
    if case["call"] in ("solve", "spmv"):
        d = np.ones_like(d)
    S, A = h.spm(d)
    return h, S, A, x


def prepare(case, seed):
    h, S, A, x = _system(case, seed)
    state = {"case": case, "h": h}
    b = A @ x
    if case["call"] == "host":
        state.update(S=S, b=np.asfortranarray(b))
        return state
    state["values"] = torch.from_numpy(S.values).cuda()
    if case["call"] == "spmv":
        state.update(x=torch.from_numpy(np.ascontiguousarray(x[:, 0])).cuda(),
                     b=torch.from_numpy(np.random.default_rng(seed).standard_normal(x.shape[0])).cuda())
    elif case["call"] == "adjoint":
        g = A.T @ x[:, 1]
        state.update(b=torch.from_numpy(b[:, 0].copy()).cuda().requires_grad_(True),
                     g=torch.from_numpy(g).cuda())
        state["values"].requires_grad_(True)
    else:
        B = torch.from_numpy(np.ascontiguousarray(b.T)).cuda()
        state["b"] = B[0].clone() if case["nrhs"] == 1 else B.t()
    if case["call"] in ("solve", "spmv") and not h.factored:
        px.numfact_device(h.pd, state["values"])
        h.factored = True
    return state


def run(state):
    case, pd = state["case"], state["h"].pd
    call = case["call"]
    if call == "factor_solve":
        px.numfact_device(pd, state["values"])
    if call in ("factor_solve", "solve"):
        x = state["b"].clone()
        px.solve_device(pd, x)
        return x
    if call == "factor_refine":
        px.numfact_device(pd, state["values"])
        x = torch.empty_like(state["b"])
        px.solve_refine_device(pd, state["b"], x)
        return x
    if call == "host":
        px.task_numfact(pd, state["S"])
        x = state["b"].copy(order="F")
        px.task_solve(pd, state["S"], x)
        return x
    if call == "adjoint":
        x = diff_solve(state["values"], state["b"], state["h"].solver)
        gv, gb = torch.autograd.grad(x, (state["values"], state["b"]), state["g"])
        return {"x": x.detach(), "grad_values": gv, "grad_b": gb}
    r = state["b"].clone()
    px.spmv_device(pd, -1.0, state["x"], 1.0, r)
    return r


def exact(case, seed):
    """The drawn solution itself (cond(A) * 1e-16 from the solution of the rounded system)."""
    if case["call"] not in ("adjoint", "spmv"):
        x = _truth(case, seed)[1]
        return x[:, 0].copy() if case["nrhs"] == 1 and case["call"] != "host" else x
    h, S, A, x = _system(case, seed)
    if case["call"] == "spmv":
        return np.random.default_rng(seed).standard_normal(x.shape[0]) - A @ x[:, 0]
    x, lam = x[:, 0], x[:, 1]
    rows, cols = S.rowptr, np.repeat(np.arange(S.n), np.diff(S.colptr))  # the stored (lower) triangle
    gv = -(lam[rows] * x[cols] + np.where(rows == cols, 0.0, lam[cols] * x[rows]))
    return {"x": x.copy(), "grad_values": gv, "grad_b": lam.copy()}


_structure = {}


def _size(case):
    """n, stored entries, factor entries and factorization flops of the analysed pattern."""
    key = _key(case)
    if key not in _structure:
        h = _handle(case)
        i = px.solver_info(h.pd)
        lu = case["fact"] == "GETRF"
        nnz = h.A.nnz if lu else (h.A.nnz + i["n"]) // 2
        _structure[key] = (i["n"], nnz, h.A.nnz, i["coefnbr"] * (2 if lu else 1), i["thflops"])
    return _structure[key]


def work(case):
    """A factorization reads the values and writes the factor; a triangular solve reads the factor once per sweep
    (half of a symmetric or unsymmetric pair each way) and the right-hand sides; both are bound by these."""
    n, nnz, full, coef, flops = _size(case)
    es, k = (4 if case["mixed"] else 8), case["nrhs"]
    if case["call"] == "spmv":  # values and 32-bit columns of the whole matrix, row pointers, x, b and r
        return {"bytes": 12 * full + 4 * (n + 1) + 24 * n, "flops": 2 * full}
    sweeps = es * coef * (1 if case["fact"] == "GETRF" else 2) + 16 * n * k
    sflops = 2 * coef * k * (1 if case["fact"] == "GETRF" else 2)
    if case["call"] == "solve":
        return {"bytes": sweeps, "flops": sflops}
    if case["call"] == "adjoint":  # factorization, two solves, the gradient over the pattern
        return {"bytes": 8 * nnz + es * coef + 2 * sweeps + 24 * nnz, "flops": flops + 2 * sflops + 4 * nnz}
    return {"bytes": 8 * nnz + es * coef + sweeps, "flops": flops + sflops}


# Largest relative difference of the solutions of correct implementations, a few times what two runs (whose scattered
# sums are ordered differently) and the drawn solution differ by: FP64 factors, FP64 refinement of FP32 factors to the
# stopping test, one application of FP32 factors.  The shifted elastic matrix is close to singular.
REL = {"lap": (1e-13, 1e-9, 1e-5), "cd": (1e-13, 1e-11, 1e-5), "grf": (2e-12, 1e-9, 1e-3), "el": (1e-10, 1e-10, 1e-2)}


def tolerance(case):
    """cond(A) times the roundoff of the factors; refined solutions: cond(A) times the stopping test's 1e-12."""
    if case["call"] == "spmv":
        return {"rel": 1e-15, "max": 1e-14}
    i = 0 if not case["mixed"] else 1 if case["call"] == "factor_refine" else 2
    return {"rel": REL[case["matrix"]][i]}
