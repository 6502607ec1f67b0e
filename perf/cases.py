"""Timed cases of the solver path: what a program that uses this package has it do.

Multigrid solves from the smallest served grid to the largest one, the mixed-precision
refinement, a batch of systems of different sizes, the two conjugate-gradient solvers,
the legacy banded multigrid, and the single operators that such programs call on their
own (smoother, defect with its norm, ELL and CSR products).  All right-hand sides are
b = A u* with u* uniform on [-1, 1), so the solution of a solve is known; b is formed
with plain torch operations, not with the package's kernels.
"""
import math

import numpy as np
import torch

import honei_b200 as hb
from honei_b200.inputs import q1_coefficient_operator

DEV = "cuda"
F64, F32 = torch.float64, torch.float32


# ---- the cases ---------------------------------------------------------------------------

def listed():
    return [
        # one request of the smallest served size class: latency and launches
        {"name": "mg_level6", "kind": "mg", "level": 6, "pre": 4, "post": 4, "eps": 1e-8, "exact_cg": False},
        # the benchmark's single-system solves: one and four million unknowns, V(4,4) to 1e-10
        {"name": "mg_level10", "kind": "mg", "level": 10, "pre": 4, "post": 4, "eps": 1e-10, "exact_cg": False},
        {"name": "mg_level11", "kind": "mg", "level": 11, "pre": 4, "post": 4, "eps": 1e-10, "exact_cg": False},
        # the same system by FP64 refinement around FP32 multigrid
        {"name": "refine_level11", "kind": "refine", "level": 11, "pre": 4, "post": 4, "eps": 1e-10},
        # a quarter of the benchmark's batch: many small and middle systems, some with 8 right-hand sides
        {"name": "batch_128", "kind": "batch", "systems": 128, "lo": 4, "hi": 9, "mix": 2024, "eps": 1e-8},
        # unpreconditioned CG on one small grid, to 1e-8: a chain of some 400 dependent steps
        {"name": "cg_level7", "kind": "cg", "level": 7, "eps": 1e-8},
        # Jacobi-preconditioned CG on an operator whose rows all differ, an odd number of cells, 200 steps
        {"name": "pcg_cells700", "kind": "pcg", "cells": 700, "steps": 200},
        # the legacy multigrid on nine stored bands (levels 1..9), V(2,2) to 1e-8
        {"name": "banded_mg_level9", "kind": "banded", "level": 9, "smooth": 2, "eps": 1e-8},
        # a smoother call of a program that builds its own cycle, single precision
        {"name": "smoother_level10_f32", "kind": "smooth", "level": 10, "sweeps": 4, "dtype": "f32"},
        # the convergence check of such a program: defect and its squared norm, largest grid
        {"name": "defect_level11_f64", "kind": "defect", "level": 11, "dtype": "f64"},
        # a product with a general ELL matrix, ragged size
        {"name": "ell_product_cells1000_f64", "kind": "ell", "cells": 1000, "dtype": "f64"},
        # a product with a CSR matrix of ragged rows, a few of them long
        {"name": "csr_product_300k_f32", "kind": "csr", "rows": 300007, "mean": 24, "long": 12, "dtype": "f32"},
    ]


def draw(rng):
    kind = rng.choice(["mg", "mg", "mg", "refine", "refine", "batch", "cg", "pcg", "banded", "smooth", "defect", "ell",
                       "csr"])
    log_int = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if kind in ("mg", "refine"):
        pre, post = rng.choice([(4, 4), (4, 4), (2, 2), (3, 3), (2, 4), (5, 3)])
        c = {"kind": kind, "level": rng.randint(5, 11), "pre": pre, "post": post, "eps": rng.choice([1e-8, 1e-9, 1e-10])}
        if kind == "mg":
            c["exact_cg"] = rng.random() < 0.25
        return c
    if kind == "batch":
        lo = rng.randint(4, 7)
        hi = rng.randint(lo, 9)
        return {"kind": kind, "systems": log_int(4, 128), "lo": lo, "hi": hi, "mix": rng.randrange(1 << 20),
                "eps": rng.choice([1e-8, 1e-9])}
    if kind == "cg":
        return {"kind": kind, "level": rng.randint(4, 8), "eps": rng.choice([1e-6, 1e-7, 1e-8])}
    if kind == "pcg":
        return {"kind": kind, "cells": log_int(150, 900), "steps": rng.randint(50, 200)}
    if kind == "banded":
        return {"kind": kind, "level": rng.randint(5, 10), "smooth": rng.choice([2, 2, 4]), "eps": rng.choice([1e-6, 1e-8])}
    dt = rng.choice(["f64", "f32"])
    if kind == "smooth":
        return {"kind": kind, "level": rng.randint(6, 11), "sweeps": rng.randint(1, 6), "dtype": dt}
    if kind == "defect":
        return {"kind": kind, "level": rng.randint(7, 11), "dtype": dt}
    if kind == "ell":
        return {"kind": kind, "cells": log_int(100, 1100), "dtype": dt}
    return {"kind": "csr", "rows": log_int(5000, 320000), "mean": rng.randint(6, 28), "long": rng.randint(0, 16), "dtype": dt}


# ---- inputs ------------------------------------------------------------------------------

def _dtype(case):
    return F32 if case["dtype"] == "f32" else F64


def _uniform(n, seed, dtype=F64):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.rand(n, generator=g, dtype=F64, device=DEV).mul_(2.0).sub_(1.0).to(dtype)


def _nodes(level):
    return (1 << level) + 1


def _q1_apply(u, m):
    """The constant-coefficient Q1 operator: 8/3 and -1/3 inside, unit rows on the boundary."""
    v = u.reshape(m, m)
    out = v.clone()
    s = v[:, :-2] + v[:, 1:-1] + v[:, 2:]
    c = v[1:-1, 1:-1]
    ring = s[:-2] + s[1:-1] + s[2:] - c
    out[1:-1, 1:-1] = (8.0 / 3.0) * c - ring / 3.0
    return out.reshape(-1)


def _coefficients(cells, seed):
    """Per-cell diffusion coefficients, contrast 4."""
    return np.power(4.0, np.random.default_rng(seed).uniform(-0.5, 0.5, (cells, cells)))


def _coefficient_operator(cells, seed, npdt):
    """The package's input layout of the variable-coefficient operator."""
    return q1_coefficient_operator(_coefficients(cells, seed), npdt)


def _ell_apply(op, x):
    """An ELL product in 64 bits from its arrays, slot after slot (padding slots hold zeros)."""
    rows, _, stride, K, Aj, Ax, _ = op
    aj, ax = Aj.reshape(K, stride).astype(np.int64), Ax.reshape(K, stride)
    y = torch.zeros(rows, dtype=F64, device=DEV)
    for k in range(K):
        y += torch.from_numpy(ax[k, :rows].astype(np.float64)).to(DEV) * x[torch.from_numpy(aj[k, :rows]).to(DEV)]
    return y


def _batch_systems(case):
    r = np.random.default_rng(case["mix"])
    n = case["systems"]
    levels = r.integers(case["lo"], case["hi"] + 1, n)
    nrhs = np.ones(n, np.int64)
    nrhs[r.permutation(n)[:n // 4]] = 8
    return [(int(l), int(k)) for l, k in zip(levels, nrhs)]


def _csr_arrays(case, seed):
    r = np.random.default_rng(seed)
    n, mean = case["rows"], case["mean"]
    length = r.integers(1, 2 * mean, n)
    length[r.permutation(n)[:case["long"]]] = min(n // 2, 2000)
    ar = np.zeros(n + 1, np.int64)
    np.cumsum(length, out=ar[1:])
    nnz = int(ar[-1])
    row = np.repeat(np.arange(n), length)
    aj = (row + r.integers(-1500, 1501, nnz)) % n           # near the diagonal, as in a mesh matrix
    ax = r.uniform(-1.0, 1.0, nnz).astype(np.float32 if case["dtype"] == "f32" else np.float64)
    return ar, aj, ax, row


def _solution(case, seed):
    kind = case["kind"]
    if kind == "pcg":
        return _uniform((case["cells"] + 1) ** 2, seed)
    return _uniform(_nodes(case["level"]) ** 2, seed)


def prepare(case, seed):
    kind = case["kind"]
    V = hb.DenseVector
    if kind in ("mg", "refine", "cg", "banded"):
        level = case["level"]
        m = _nodes(level)
        b = V(_q1_apply(_solution(case, seed), m))
        s = {"kind": kind, "case": case, "b": b, "x": V(m * m)}
        if kind == "mg":
            s["mg"] = hb.MGData.poisson_q1(3, level, params=hb.mg_params(
                case["pre"], case["post"], eps=case["eps"], coarse_exact=case["exact_cg"]))
        elif kind == "refine":
            s["A"] = hb.SparseMatrixELL.poisson_q1(level)
            s["mg"] = hb.MGData.poisson_q1(3, level, dtype=F32, params=hb.mg_params(
                case["pre"], case["post"], eps=1e-3, coarse_eps=1e-3, coarse_exact=False, coarse_fp64=True))
        elif kind == "cg":
            s["A"] = hb.SparseMatrixELL.poisson_q1(level)
        else:
            A = [hb.BandedMatrixQx.poisson_q1(l) for l in range(1, level + 1)]
            s["mg"] = hb.Multigrid(A, 1, hb.mg_info(n_max_iter=100, tolerance=case["eps"], n_pre_smooth=case["smooth"]))
        return s
    if kind == "batch":
        systems = _batch_systems(case)
        bs, sizes = [], []
        for i, (level, k) in enumerate(systems):
            m = _nodes(level)
            u = _uniform(k * m * m, seed * 1009 + i).reshape(k, m * m)
            bs.append(torch.stack([_q1_apply(u[j], m) for j in range(k)]))
            sizes.append(k * m * m)
        flat = torch.empty(sum(sizes), dtype=F64, device=DEV)
        return {"kind": kind, "case": case, "solver": hb.BatchedPoissonSolver(
            systems, params=hb.batch_params(eps=case["eps"])), "b": bs, "flat": flat,
                "x": list(torch.split(flat, sizes))}
    if kind == "pcg":
        op = _coefficient_operator(case["cells"], seed, np.float64)
        A = hb.SparseMatrixELL.from_arrays(*op)
        P = hb.RISmoother.jacobi_precon(A, 1.0)
        return {"kind": kind, "case": case, "solver": hb.KrylovSolver(hb.HB2_CG_VAR, A, P, case["steps"], 0.0),
                "b": V(_ell_apply(op, _solution(case, seed))), "x": V(A.rows())}
    dt = _dtype(case)
    if kind in ("smooth", "defect"):
        m = _nodes(case["level"])
        A = hb.SparseMatrixELL.poisson_q1(case["level"], dt)
        b = V(_q1_apply(_uniform(m * m, seed), m).to(dt))
        x = V(_uniform(m * m, seed + 500009, dt))
        if kind == "smooth":
            return {"kind": kind, "case": case, "A": A, "P": hb.RISmoother.jacobi_precon(A, 0.7), "b": b, "x0": x,
                    "x": x.copy(), "t": V(m * m, dtype=dt)}
        return {"kind": kind, "case": case, "A": A, "b": b, "x": x, "r": V(m * m, dtype=dt),
                "norm2": torch.zeros(1, dtype=F64, device=DEV)}
    if kind == "ell":
        A = hb.SparseMatrixELL.from_arrays(*_coefficient_operator(
            case["cells"], seed, np.float32 if dt == F32 else np.float64))
    else:
        ar, aj, ax, _ = _csr_arrays(case, seed)
        A = hb.SparseMatrixCSR.from_arrays(case["rows"], case["rows"], ar, aj, ax)
    return {"kind": kind, "case": case, "A": A, "x": V(_uniform(A.columns(), seed + 500009, dt)), "y": V(A.rows(), dtype=dt)}


# ---- one pass ----------------------------------------------------------------------------

def run(s):
    kind, case = s["kind"], s["case"]
    if kind == "mg":
        hb.fill(s["x"], 0.0)
        return hb.MGSolver.value(s["mg"], s["b"], s["x"]).elements
    if kind == "refine":
        hb.fill(s["x"], 0.0)
        return hb.IRSolver.value(s["A"], s["b"], s["x"], s["mg"], eps=case["eps"], reset_inner=True)[0].elements
    if kind == "batch":
        B = s["solver"]
        for i, b in enumerate(s["b"]):
            B.set_rhs(i, b)
        B.solve()
        for i, x in enumerate(s["x"]):
            B.solution(i, out=x)
        return s["flat"]                                  # all solutions, one after the other
    if kind == "cg":
        hb.fill(s["x"], 0.0)
        return hb.CGSolver.value(s["A"], None, s["b"], s["x"], 5000, eps_relative=case["eps"])[0].elements
    if kind == "pcg":
        hb.fill(s["x"], 0.0)
        return s["solver"].solve(s["b"], s["x"])[0].elements
    if kind == "banded":
        hb.fill(s["x"], 0.0)
        return s["mg"].value(s["b"], s["x"])[0].elements
    if kind == "smooth":
        hb.copy(s["x0"], s["x"])
        return hb.RISmoother.value(s["A"], s["P"], s["b"], s["x"], temps=[s["t"]], max_iters=case["sweeps"]).elements
    if kind == "defect":
        return hb.Defect.value(s["r"], s["b"], s["A"], s["x"], norm2_out=s["norm2"]).elements, s["norm2"]
    return hb.Product.value(s["y"], s["A"], s["x"]).elements


# ---- what a pass cannot do without -------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("mg", "refine", "banded"):
        # b in, x out; about eight cycles of the smoothing steps, a defect each way and the
        # transfers, on levels whose sizes fall by four; a nine-point row is 17 operations
        n = _nodes(case["level"]) ** 2
        steps = 2 * case["smooth"] + 2 if kind == "banded" else case["pre"] + case["post"] + 2
        bands = 9 * 8 * n * 4 // 3 if kind == "banded" else 0
        return {"bytes": 16 * n + bands, "flops": 8 * steps * 20 * n * 4 // 3}
    if kind == "batch":
        n = sum(k * _nodes(l) ** 2 for l, k in _batch_systems(case))
        return {"bytes": 16 * n, "flops": 8 * (11 * 20 * 4 // 3 + 30) * n}
    if kind == "cg":
        n = _nodes(case["level"]) ** 2
        steps = 3 * (1 << case["level"])
        return {"bytes": 16 * n, "flops": steps * 27 * n}
    if kind == "pcg":
        n = (case["cells"] + 1) ** 2
        return {"bytes": 9 * 8 * n + 24 * n, "flops": case["steps"] * 30 * n}
    s = 4 if case["dtype"] == "f32" else 8
    if kind in ("smooth", "defect"):
        n = _nodes(case["level"]) ** 2
        if kind == "smooth":
            return {"bytes": 5 * s * n, "flops": case["sweeps"] * 20 * n}      # x0, b, P in; x out, written once more
        return {"bytes": 3 * s * n, "flops": 20 * n}
    if kind == "ell":
        n = (case["cells"] + 1) ** 2
        return {"bytes": (9 * (s + 4) + 2 * s) * n, "flops": 18 * n}
    nnz = case["rows"] * case["mean"] + 2000 * case["long"]
    return {"bytes": nnz * (s + 4) + case["rows"] * (2 * s + 4), "flops": 2 * nnz}


def tolerance(case):
    """About four times the largest difference measured between two orders of the sums."""
    kind = case["kind"]
    if kind == "mg":          # coarsest CG with sequential against tree-ordered dots: up to 6.7e-9
        return {"rel": 3e-8}
    if kind == "refine":      # coarsest CG's dots 3.5e-7, its precision 2.4e-6: the FP32 cycles decide the last digits
        return {"rel": 1e-5}
    if kind == "batch":       # right-hand sides changed by less than FP32 rounding (2e-8): up to 2.1e-6
        return {"rel": 8e-6}
    if kind == "cg":          # one step more or less at the stopping test, see _CG_STEP
        return {"rel": _CG_STEP * case["eps"]}
    if kind == "pcg":         # right-hand side changed by one unit in the last place: up to 1.1e-14
        return {"rel": 5e-14}
    if kind == "banded":      # the same: up to 3.7e-14
        return {"rel": 2e-13}
    if kind == "smooth":      # against 64 bits 6.1e-8; FP64 1.3e-16
        return {"rel": 2.5e-7 if case["dtype"] == "f32" else 6e-16}
    # products and defects against 64 bits: FP32 up to 1.5e-7, FP64 up to 1.9e-16
    return {"rel": 6e-7 if case["dtype"] == "f32" else 8e-16}


# the last step of unpreconditioned CG changes the solution by 2.5 to 7.1 times eps (levels 4 to 8)
_CG_STEP = 28.0


# ---- 64-bit values -----------------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind in ("mg", "refine", "cg", "banded"):
        return _solution(case, seed)                      # the solves approach u*
    if kind == "batch":
        return torch.cat([_uniform(k * _nodes(l) ** 2, seed * 1009 + i) for i, (l, k) in
                          enumerate(_batch_systems(case))])
    if kind == "pcg":
        return _pcg_exact(case, seed)
    if kind in ("smooth", "defect"):
        dt = _dtype(case)
        m = _nodes(case["level"])
        b = _q1_apply(_uniform(m * m, seed), m).to(dt).to(F64)
        x = _uniform(m * m, seed + 500009, dt).to(F64)
        # the matrix entries as the operator's type holds them
        v = torch.tensor([8.0 / 3.0, -1.0 / 3.0], dtype=F64).to(dt).to(F64).tolist()

        def apply(u):
            g = u.reshape(m, m)
            out = g.clone()
            t = g[:, :-2] + g[:, 1:-1] + g[:, 2:]
            c = g[1:-1, 1:-1]
            out[1:-1, 1:-1] = v[0] * c + v[1] * (t[:-2] + t[1:-1] + t[2:] - c)
            return out.reshape(-1)
        if kind == "defect":
            r = b - apply(x)
            return r, (r * r).sum().reshape(1)
        P = torch.full((m, m), 0.7, dtype=F64, device=DEV)
        P[1:-1, 1:-1] = 0.7 / v[0]
        P = P.to(dt).to(F64).reshape(-1)
        for _ in range(case["sweeps"]):
            x = x + P * (b - apply(x))
        return x
    x = None
    if kind == "ell":
        op = _coefficient_operator(case["cells"], seed, np.float32 if case["dtype"] == "f32" else np.float64)
        x = _uniform(op[1], seed + 500009, _dtype(case)).to(F64)
        return _ell_apply(op, x)
    ar, aj, ax, row = _csr_arrays(case, seed)
    x = _uniform(case["rows"], seed + 500009, _dtype(case)).to(F64).cpu().numpy()
    return torch.from_numpy(np.add.reduceat(ax.astype(np.float64) * x[aj], ar[:-1]))


def _pcg_exact(case, seed):
    """The same number of preconditioned steps in 64 bits from x = 0."""
    op = _coefficient_operator(case["cells"], seed, np.float64)
    rows, _, stride, K, Aj, Ax, _ = op
    aj = [torch.from_numpy(c.astype(np.int64)).to(DEV) for c in Aj.reshape(K, stride)]
    ax = [torch.from_numpy(c).to(DEV) for c in Ax.reshape(K, stride)]

    def apply(u):
        y = ax[0] * u[aj[0]]
        for k in range(1, K):
            y += ax[k] * u[aj[k]]
        return y
    diag = torch.ones(rows, dtype=F64, device=DEV)
    idx = torch.arange(rows, device=DEV)
    for k in range(K):
        hit = (aj[k] == idx) & (ax[k] != 0)
        diag = torch.where(hit, ax[k], diag)
    b = apply(_solution(case, seed))
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rho = torch.dot(r, z)
    for _ in range(case["steps"]):
        v = apply(p)
        a = rho / torch.dot(v, p)
        x += a * p
        r -= a * v
        z = r / diag
        new = torch.dot(r, z)
        p = z + (new / rho) * p
        rho = new
    return x
