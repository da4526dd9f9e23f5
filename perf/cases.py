"""Workloads of the sparse-direct solver, each through the public entry points.

A case is a dict of plain values:

``kind``       "step"      new values of A -> LDL -> solve (the plan and the
                           analysis are kept, as a frequency sweep, a Newton
                           loop or a time stepper keeps them),
               "solve"     a solve over stored factors,
               "batch"     many independent 2D problems in one plan,
               "gradient"  forward and backward of the differentiable solve.
``operator``   "laplacian" real 7-point (5-point) operator + shift,
               "magnetic"  its Hermitian form with a phase on every coupling,
               "helmholtz" complex-symmetric Helmholtz with a PML and a
                           heterogeneous velocity, 10 points per wavelength.
``precision``  "double": FP64 fronts, plain solve; "single": FP32 fronts and
               refinement in FP64 to a relative residual of 1e-10.
``front``      the front type LDL is asked for.
``ordering``   "natural" or "graph" nested dissection.
``diag``       the Laplacian's diagonal; below 6 (below 4 in 2D) the operator
               is indefinite, as in shift-invert iterations.

Values, right-hand sides and cotangents come from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import clique_b200 as cliq
from clique_b200 import operators as ops

TOL = 1e-10
PHASE = 0.4


def _step(name, operator, nx, ny, nz, nrhs, precision, front="LDL_2D", ordering="natural", cutoff=128, diag=6.1,
          kind="step"):
    c = {"kind": kind, "operator": operator, "nx": nx, "ny": ny, "nz": nz, "nrhs": nrhs, "precision": precision,
         "front": front, "ordering": ordering, "cutoff": cutoff}
    if operator != "helmholtz":
        c["diag"] = diag
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest factor + solve: a coarse-grid or subdomain solver called
        # over and over, where launches and latency count
        _step("lap12_fp64", "laplacian", 12, 11, 9, 1, "double", cutoff=48),
        # the plain FP64 operator of the configurations: 27,000 unknowns
        _step("lap30_fp64", "laplacian", 30, 30, 30, 1, "double"),
        # a 2D field problem with ragged sides: many small fronts, deep tree
        _step("lap2d_701x503_fp64", "laplacian", 701, 503, 1, 3, "double", diag=4.1),
        # plain FP64 complex factor + solve at the size of the gradient workload
        _step("helm64_fp64", "helmholtz", 64, 64, 64, 1, "double"),
        # the headline: 100^3 Helmholtz, FP32 fronts, refinement, 4 sources
        _step("helm100_fp32", "helmholtz", 100, 100, 100, 4, "single"),
        # the large real configuration scaled to one state of a few GB: many
        # right-hand sides, ragged sides, leaf cutoff 256
        _step("lap101x99x90_fp32", "laplacian", 101, 99, 90, 16, "single", cutoff=256),
        # Hermitian indefinite operator with pivoting inside the fronts, FP64
        _step("mag40_pivot_fp64", "magnetic", 40, 37, 33, 2, "double", front="LDL_INTRAPIV_2D", diag=5.0),
        # complex symmetric with pivoting, FP32 fronts and refinement
        _step("helm48_pivot_fp32", "helmholtz", 48, 48, 48, 4, "single", front="LDL_INTRAPIV_2D"),
        # what the black-box solve does by default: graph ordering, pivoting
        _step("lap_graph_pivot_fp64", "laplacian", 29, 27, 23, 1, "double", front="LDL_INTRAPIV_1D", ordering="graph",
              diag=5.5),
        # factor once, solve many: one stored-factor solve of a few columns
        _step("stored_helm56_fp64", "helmholtz", 56, 56, 56, 8, "double", kind="solve"),
        # a survey of independent 2D problems of uneven size in one plan
        {"name": "batch64_fp32", "kind": "batch", "count": 64, "lo": 32, "hi": 96, "rhs_hi": 8, "cutoff": 64},
        # one inversion step: forward solve and gradient over the same factors
        {"name": "gradient40_fp32", "kind": "gradient", "nx": 40, "ny": 40, "nz": 40, "nrhs": 1, "precision": "single",
         "cutoff": 128},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi):
    """Three sides around one log-uniform size, ragged as often as not."""
    a = _logint(rng, lo, hi)
    if rng.random() < 0.4:
        return a, a, a
    return tuple(max(4, min(hi, int(a * rng.uniform(0.75, 1.15)))) for _ in range(3))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "pivot", "pivot", "solve", "batch", "gradient"])
    cutoff = rng.choice([48, 64, 128, 128, 256])
    if kind == "batch":
        lo = rng.randint(20, 40)
        return {"kind": "batch", "count": _logint(rng, 8, 72), "lo": lo, "hi": lo + rng.randint(8, 56),
                "rhs_hi": _logint(rng, 1, 16), "cutoff": rng.choice([48, 64, 128])}
    if kind == "gradient":
        nx, ny, nz = _sides(rng, 12, 44)
        return {"kind": "gradient", "nx": nx, "ny": ny, "nz": nz, "nrhs": rng.choice([1, 1, 2, 5]),
                "precision": rng.choice(["single", "double"]), "cutoff": cutoff}
    precision = rng.choice(["single", "double"])
    nrhs = _logint(rng, 1, 24)
    if kind == "pivot":
        operator = rng.choice(["laplacian", "magnetic", "helmholtz"])
        nx, ny, nz = _sides(rng, 9, 48)
        return _step(None, operator, nx, ny, nz, nrhs, precision, front=rng.choice(["LDL_INTRAPIV_1D", "LDL_INTRAPIV_2D"]),
                     ordering=rng.choice(["natural", "graph"]) if nx * ny * nz < 30000 else "natural", cutoff=cutoff,
                     diag=round(rng.uniform(5.0, 6.2), 3))
    operator = rng.choice(["laplacian", "laplacian", "magnetic", "helmholtz", "helmholtz"])
    if operator != "helmholtz" and rng.random() < 0.3:
        nx, ny = _logint(rng, 40, 700), _logint(rng, 40, 700)
        return _step(None, operator, nx, ny, 1, nrhs, precision, cutoff=cutoff, diag=4.1,
                     kind=kind if rng.random() < 0.7 else "solve")
    nx, ny, nz = _sides(rng, 9, 60 if precision == "double" else 84)
    front = rng.choice(["LDL_2D", "BLOCK_LDL_2D"]) if kind == "solve" else rng.choice(["LDL_1D", "LDL_2D"])
    if front == "BLOCK_LDL_2D":
        nx, ny, nz = min(nx, 48), min(ny, 48), min(nz, 48)
    return _step(None, operator, nx, ny, nz, nrhs, precision, front=front, cutoff=cutoff, kind=kind)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _operator(case, seed):
    """A as CSR."""
    dims = case["nx"], case["ny"], case["nz"]
    if case.get("operator", "helmholtz") == "helmholtz":
        vel = ops.smooth_velocity(dims, seed)
        h = 1.0 / (dims[0] + 1)
        omega = ops.omega_for_ppw(dims[0], float(vel.min()))
        return ops.helmholtz_pml_3d(*dims, omega, vel, L=tuple((d + 1) * h for d in dims))
    diag = case["diag"] + _shift(seed)
    A = ops.laplacian_3d(*dims, diag) if dims[2] > 1 else ops.laplacian_2d(dims[0], dims[1], diag)
    if case["operator"] == "magnetic":
        step = np.sign(A.colind - np.repeat(np.arange(A.n), np.diff(A.rowptr)))
        A.values = A.values * np.exp(1j * PHASE * step)
    return A


def _shift(seed):
    """The diagonal moves a little with the seed (the real configuration's 0.1 stays the centre)."""
    return 0.02 * (np.random.default_rng(seed).random() - 0.5)


def _rhs(case, seed, n, cplx):
    return ops.random_rhs(n, case["nrhs"], seed=seed + 1, complex_=cplx)


def _column_major(B):
    """Device copy, column-major (n, nrhs)."""
    return torch.from_numpy(np.ascontiguousarray(B.T)).cuda().t()


def _order(case, A):
    if case["ordering"] == "graph":
        return cliq.NestedDissection(A, case["cutoff"])
    return cliq.NaturalNestedDissection(case["nx"], case["ny"], case["nz"], A, case["cutoff"])


def _batch_problems(case, seed):
    rng = np.random.default_rng(seed)
    sides = [int(s) for s in np.linspace(case["lo"], case["hi"], case["count"]).round()]
    sides = [sides[i] for i in rng.permutation(case["count"])]
    nrhs = 1 + np.arange(case["count"]) % case["rhs_hi"]
    mats = [ops.helmholtz_workload_2d(s, seed=seed * 1009 + i)[0] for i, s in enumerate(sides)]
    B = np.zeros((sum(A.n for A in mats), case["rhs_hi"]), np.complex128)
    r0 = 0
    for i, A in enumerate(mats):
        B[r0:r0 + A.n, :nrhs[i]] = ops.random_rhs(A.n, int(nrhs[i]), seed=seed * 1013 + i, complex_=True)
        r0 += A.n
    return mats, sides, B


def prepare(case, seed):
    if case["kind"] == "batch":
        from clique_b200.batch import BatchSolver
        mats, sides, B = _batch_problems(case, seed)
        solver = BatchSolver(mats, [(s, s, 1) for s in sides], cutoff=case["cutoff"], precision="single")
        return {"case": case, "solver": solver, "values": torch.from_numpy(solver.A.values).cuda(), "B": _column_major(B)}
    A = _operator(case, seed)
    values = torch.from_numpy(A.values).cuda()
    B = _column_major(_rhs(case, seed, A.n, A.is_complex))
    if case["kind"] == "gradient":
        from clique_b200.autograd import SparseLDLSolver
        solver = SparseLDLSolver(A, (case["nx"], case["ny"], case["nz"]), cutoff=case["cutoff"],
                                 precision=case["precision"])
        G = _column_major(ops.random_rhs(A.n, case["nrhs"], seed=seed + 2, complex_=True))
        return {"case": case, "solver": solver, "values": values.requires_grad_(), "B": B.requires_grad_(), "G": G}
    map_, sep, info = _order(case, A)
    L = cliq.DistSymmFrontTree(A, map_, sep, info, case["operator"] == "magnetic", precision=case["precision"],
                               keep_matrix=True, stream=torch.cuda.current_stream().cuda_stream)
    state = {"case": case, "info": info, "L": L, "values": values, "B": B,
             "front": getattr(cliq.SymmFrontType, case["front"])}
    if case["kind"] == "solve":
        cliq.LDL(info, L, state["front"])
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        X, _, _ = state["solver"].run(state["values"], state["B"], tol=TOL)
        return X
    if case["kind"] == "gradient":
        from clique_b200.autograd import sparse_solve
        X = sparse_solve(state["values"], state["B"], state["solver"])
        gvalues, gB = torch.autograd.grad(X, (state["values"], state["B"]), state["G"])
        return {"X": X.detach(), "gvalues": gvalues.resolve_conj(), "gB": gB.resolve_conj()}
    L, info = state["L"], state["info"]
    if case["kind"] == "step":
        L.Initialize(state["values"])
        cliq.LDL(info, L, state["front"])
    if case["precision"] == "single":
        X, _, _ = cliq.RefinedSolve(L, state["B"], TOL)
        return X
    return cliq.Solve(info, L, state["B"].clone())


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _tree_work(info):
    """(flops of a real LDL^T, stored entries of the factors) of an analysis."""
    flops = entries = 0.0
    for node in info.localNodes:
        n, u = float(node.size), float(len(node.lowerStruct))
        flops += n ** 3 / 3 + u * n * n + u * u * n
        entries += n * (n + 1) / 2 + u * n
    return flops, entries


def work(case):
    """Bytes: the values and the right-hand sides read, the solution written,
    the factors written (a step) or read (a solve) once.  Flops: the
    factorization and one forward and backward sweep per right-hand side."""
    if case["kind"] == "batch":
        mats, sides, B = _batch_problems(case, 0)
        flops = entries = nnz = 0.0
        for A, s in zip(mats, sides):
            f, e = _tree_work(cliq.NaturalNestedDissection(s, s, 1, A, case["cutoff"])[2])
            nrhs = (np.abs(B[:1]) > 0).sum()
            flops, entries, nnz = flops + 4 * f + 16 * e * nrhs, entries + e, nnz + A.nnz
            B = B[A.n:]
        n, k = sum(A.n for A in mats), case["rhs_hi"]
        return {"bytes": 16 * nnz + 8 * entries + 32.0 * n * k, "flops": float(flops)}
    A = _operator(case, 0)
    c = 4.0 if A.is_complex else 1.0
    scalar = 16 if A.is_complex else 8
    order = case if "ordering" in case else dict(case, ordering="natural")
    flops, entries = _tree_work(_order(order, A)[2])
    factor_bytes = entries * scalar / (2 if case["precision"] == "single" else 1)
    solve = 4 * c * entries * case["nrhs"]
    rhs_bytes = 2.0 * scalar * A.n * case["nrhs"]
    if case["kind"] == "solve":
        return {"bytes": factor_bytes + rhs_bytes, "flops": solve}
    if case["kind"] == "gradient":
        return {"bytes": factor_bytes + 2 * rhs_bytes + 2.0 * scalar * A.nnz, "flops": c * flops + 2 * solve}
    return {"bytes": factor_bytes + rhs_bytes + float(scalar) * A.nnz, "flops": c * flops + solve}


def tolerance(case):
    """Refined solves stop anywhere under a residual of 1e-10, which these
    operators turn into 2e-11 to 4e-10 of the solution (measured against
    ``exact``); plain FP64 solves are 1e-15 to 1.3e-11 off it, the indefinite
    ones the most, and two orders of summation differ by the same."""
    if case["kind"] == "batch" or case["precision"] == "single":
        return {"rel": 2e-9}
    return {"rel": 5e-11}


# ---------------------------------------------------------------------------
# the same in plain numpy / torch, 64 bits
# ---------------------------------------------------------------------------
def _sine(n):
    """Orthonormal sine transform (its own inverse) and the eigenvalues of the 1D chain with couplings -1."""
    j = np.arange(1, n + 1)
    return np.sqrt(2.0 / (n + 1)) * np.sin(np.pi * np.outer(j, j) / (n + 1)), -2.0 * np.cos(np.pi * j / (n + 1))


def _exact_laplacian(case, seed, B):
    dims = case["nx"], case["ny"], case["nz"]
    idx = np.arange(B.shape[0])
    x, y, z = idx % dims[0], idx // dims[0] % dims[1], idx // (dims[0] * dims[1])
    phase = np.exp(-1j * PHASE * (x + y + z))[:, None] if case["operator"] == "magnetic" else 1.0
    V = (np.conj(phase) * B).reshape(dims[2], dims[1], dims[0], -1)
    (Q1, e1), (Q2, e2), (Q3, e3) = _sine(dims[0]), _sine(dims[1]), _sine(dims[2])
    if dims[2] == 1:
        e3 = np.zeros(1)

    def transform(V):
        return np.einsum("ac,zycr->zyar", Q1, np.einsum("by,zyxr->zbxr", Q2, np.einsum("cz,zyxr->cyxr", Q3, V,
                         optimize=True), optimize=True), optimize=True)

    lam = case["diag"] + _shift(seed) + e3[:, None, None] + e2[None, :, None] + e1[None, None, :]
    return phase * transform(transform(V) / lam[..., None]).reshape(B.shape)


class _Planes:
    """Block elimination of a grid operator plane by plane (line by line in
    2D), pivoting inside the planes, with two steps of refinement."""

    def __init__(self, A, block, device):
        nb = A.n // block
        rows = np.repeat(np.arange(A.n), np.diff(A.rowptr))
        self.entries = [torch.from_numpy(v).to(device) for v in (rows, A.colind.astype(np.int64), A.values)]
        low, up = np.zeros(A.n, A.values.dtype), np.zeros(A.n, A.values.dtype)
        m = rows - A.colind == block
        low[rows[m]] = A.values[m]
        m = A.colind - rows == block
        up[rows[m]] = A.values[m]
        self.low, self.up = (torch.from_numpy(v).to(device).reshape(nb, block, 1) for v in (low, up))
        self.block, self.inv = block, []
        for k in range(nb):
            lo, hi = int(A.rowptr[k * block]), int(A.rowptr[(k + 1) * block])
            r, c, v = rows[lo:hi] - k * block, A.colind[lo:hi].astype(np.int64) - k * block, A.values[lo:hi]
            m = (c >= 0) & (c < block)
            D = torch.zeros(block, block, dtype=self.low.dtype, device=device)
            D[torch.from_numpy(r[m]).to(device), torch.from_numpy(c[m]).to(device)] = torch.from_numpy(v[m]).to(device)
            if k:
                D -= self.low[k] * self.inv[-1] * self.up[k - 1].reshape(1, block)
            self.inv.append(torch.linalg.inv(D))

    def once(self, B):
        y = list(B.reshape(-1, self.block, B.shape[1]).unbind(0))
        for k in range(1, len(y)):
            y[k] = y[k] - self.low[k] * (self.inv[k - 1] @ y[k - 1])
        y[-1] = self.inv[-1] @ y[-1]
        for k in range(len(y) - 2, -1, -1):
            y[k] = self.inv[k] @ (y[k] - self.up[k] * y[k + 1])
        return torch.cat(y)

    def solve(self, B):
        rows, cols, values = self.entries
        X = self.once(B)
        for _ in range(2):
            X = X + self.once(B.index_add(0, rows, values[:, None] * X[cols], alpha=-1))
        return X


def exact(case, seed):
    if case["kind"] == "batch":
        mats, sides, B = _batch_problems(case, seed)
        out, r0 = [], 0
        for A, s in zip(mats, sides):
            out.append(_Planes(A, s, "cpu").solve(torch.from_numpy(B[r0:r0 + A.n])))
            r0 += A.n
        return torch.cat(out)
    A = _operator(case, seed)
    B = _rhs(case, seed, A.n, A.is_complex)
    if case.get("operator", "helmholtz") != "helmholtz":
        return _exact_laplacian(case, seed, B)
    block = case["nx"] * case["ny"]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if 16.0 * block ** 3 * case["nz"] > (1e14 if device == "cuda" else 3e12):
        return None
    planes = _Planes(A, block, device)
    X = planes.solve(torch.from_numpy(B).to(device))
    if case["kind"] != "gradient":
        return X
    G = torch.from_numpy(ops.random_rhs(A.n, case["nrhs"], seed=seed + 2, complex_=True)).to(device)
    gB = planes.solve(G.conj().resolve_conj()).conj().resolve_conj()
    rows = torch.from_numpy(np.repeat(np.arange(A.n), np.diff(A.rowptr))).to(device)
    cols = torch.from_numpy(A.colind.astype(np.int64)).to(device)
    return {"X": X, "gvalues": -(gB[rows] * X[cols].conj()).sum(1), "gB": gB}
