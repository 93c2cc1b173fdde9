"""The measured work of the framework: factorizations and solves as a user's program calls them.

Every case goes through the public entry points of the package (SparseLDLT, BatchLDLT).  A case names

  op      "step"   new values into an analysed solver: factor, inertia, solve (an interior-point or time step);
          "solve"  right-hand sides against a factor that is kept;
          "batch"  many independent systems, factored and solved together from host arrays
  matrix  "laplace"  7-point Laplacian on a g^3 grid, shifted so that part of the spectrum is negative
          "kkt"      saddle point [[H, J^T], [J, 0]], H the 27-point Laplacian, J a quarter as many random rows
          "stencil"  7-point pattern with N(0, 1) values and a small diagonal: delayed pivots everywhere
  form    "fp64" the default; "tf32" / "bf16" the mixed forms with refinement; "learned" the shipped selector
  host    values and right-hand sides in numpy arrays (the reference's own interface) or already on the GPU

Values change with the seed: the Laplacian is scaled symmetrically by factors near one, the stencil and the KKT
matrix are drawn anew, and so are the right-hand sides.
"""
import functools
import importlib
import math
import os

import numpy as np
import torch

rv = importlib.import_module("rivrs-linalg_b200")

# Cost of a pass grows with the factor's operations (about g^6 for the grids, g^9 for the KKT systems, whose
# constraint rows end in one dense front): the ranges below span from where launches count to where GEMMs do.
GRID = {"laplace": (6, 80), "kkt": (6, 48), "stencil": (6, 32)}


def listed():
    return [
        # the smallest calls: a control or estimation loop that refactors a few hundred unknowns
        dict(name="laplace8_step", op="step", matrix="laplace", g=8, form="fp64", host=True, nrhs=1, mc64=False),
        # the documented example: 4,096 unknowns, 10% negative, MC64 scaling, one right-hand side
        dict(name="laplace16_step", op="step", matrix="laplace", g=16, form="fp64", host=True, nrhs=1, mc64=True),
        # general indefinite values: 2x2 pivots and delayed columns throughout
        dict(name="stencil27_step", op="step", matrix="stencil", g=27, form="fp64", host=True, nrhs=1, mc64=True),
        # an interior-point step on a middle-sized saddle point
        dict(name="kkt24_step", op="step", matrix="kkt", g=24, form="fp64", host=True, nrhs=2, mc64=True),
        # frequency-domain style: middle-sized grid, several right-hand sides
        dict(name="laplace48_step", op="step", matrix="laplace", g=48, form="fp64", host=True, nrhs=5, mc64=True),
        # a large grid with everything on the device: half a million unknowns
        dict(name="laplace80_step", op="step", matrix="laplace", g=80, form="fp64", host=False, nrhs=1, mc64=True),
        # mixed precision with refinement escalating to GMRES-IR, on the device, as the benchmark runs it
        dict(name="kkt36_bf16_step", op="step", matrix="kkt", g=36, form="bf16", host=False, nrhs=1, mc64=True),
        # the default mixed form (TF32 parts, partial sums flushed to FP64), refinement, the largest front
        dict(name="kkt45_tf32_step", op="step", matrix="kkt", g=45, form="tf32", host=False, nrhs=1, mc64=True),
        # the form chosen per front by the shipped selector
        dict(name="kkt31_learned_step", op="step", matrix="kkt", g=31, form="learned", host=True, nrhs=1, mc64=True),
        # a factor that is kept: one right-hand side at a time (time stepping, preconditioning)
        dict(name="laplace64_solve1", op="solve", matrix="laplace", g=64, form="fp64", host=False, nrhs=1, mc64=True),
        # a factor that is kept: a block of right-hand sides (sensitivities), an odd count
        dict(name="kkt36_solve13", op="solve", matrix="kkt", g=36, form="fp64", host=False, nrhs=13, mc64=True),
        # many independent systems, Laplacians and saddle points in turn, 1 to 12 right-hand sides each
        dict(name="batch8", op="batch", count=8, n_lo=1500, n_hi=20000, max_rhs=12),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "mixed", "solve", "batch"])

    def grid(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))

    if kind == "batch":
        lo = rng.randint(500, 4000)
        return dict(op="batch", count=rng.randint(2, 9), n_lo=lo, n_hi=lo + rng.randint(500, 15000),
                    max_rhs=rng.randint(1, 17))
    if kind == "mixed":
        form = rng.choice(["bf16", "tf32", "learned"])
        return dict(op="step", matrix="kkt", g=grid(18, 42), form=form, host=rng.random() < 0.5, nrhs=1, mc64=True)
    matrix = rng.choice(["laplace", "kkt", "stencil"])
    lo, hi = GRID[matrix]
    if matrix == "kkt":
        hi = 38
    nrhs = rng.choice([1, 1, 2, 3, 6, 8, 11, 17]) if kind == "solve" else rng.choice([1, 1, 1, 2, 5])
    return dict(op=kind, matrix=matrix, g=grid(lo, hi), form="fp64", host=rng.random() < 0.5, nrhs=nrhs,
                mc64=matrix != "laplace" or rng.random() < 0.5)


# ---- systems -------------------------------------------------------------------------------------------------


def _csc_columns(s):
    return np.repeat(np.arange(s.n, dtype=np.int64), np.diff(s.colptr))


@functools.lru_cache(maxsize=2)
def _laplace(g):
    return rv.problems.shifted_laplacian(g, 0.10)


def _laplace_scaling(s, seed):
    return np.exp(0.05 * np.random.default_rng([seed, 1]).standard_normal(s.n))


def _system(matrix, g, seed):
    if matrix == "kkt":
        return rv.problems.kkt(g, seed=seed)
    s = _laplace(g)
    out = rv.problems.System(name=f"{matrix}{g}", n=s.n, colptr=s.colptr, rowidx=s.rowidx, values=s.values,
                             grid=s.grid)
    row, col = s.rowidx, _csc_columns(s)
    if matrix == "laplace":
        d = _laplace_scaling(s, seed)
        out.values = s.values * (d[row] * d[col])
    else:
        # one N(0, 1) value per edge, the diagonal a tenth of that
        rng = np.random.default_rng([seed, 2])
        key = np.minimum(row, col) * np.int64(s.n) + np.maximum(row, col)
        uniq, inv = np.unique(key, return_inverse=True)
        out.values = rng.standard_normal(uniq.size)[inv]
        out.values[row == col] *= 0.1
    return out


def _batch(case, seed):
    rng = np.random.default_rng(case["count"] * 1000003 + case["n_lo"])  # sizes: the case's; values: the seed's
    systems, nrhs = [], []
    for i in range(case["count"]):
        n = math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))
        if i % 2 == 0:
            s = _system("laplace", max(4, round(n ** (1 / 3))), seed + i)
        else:
            s = _system("kkt", max(4, round((n / 1.25) ** (1 / 3))), seed + i)
        systems.append(s)
        nrhs.append(int(rng.integers(1, case["max_rhs"] + 1)))
    return systems, nrhs


def _rhs(n, nrhs, seed):
    return rv.problems.rhs_normal(n, seed=[seed, 3], nrhs=nrhs)


def _options(form):
    if form == "fp64":
        return rv.FactorOptions()
    if form == "tf32":
        return rv.FactorOptions(precision="mixed")
    return rv.FactorOptions(precision="mixed" if form == "bf16" else "learned", mixed_flush=0, mixed_operands="bf16")


# ---- preparation and passes ----------------------------------------------------------------------------------


def prepare(case, seed):
    torch.cuda.init()
    if case["op"] == "batch":
        systems, nrhs = _batch(case, seed)
        batch = rv.BatchLDLT(systems, device_budget=8 << 30)
        rhs = [_rhs(s.n, r, seed + i) for i, (s, r) in enumerate(zip(systems, nrhs))]
        return dict(op="batch", batch=batch, values=[s.values for s in systems], rhs=rhs)
    s = _system(case["matrix"], case["g"], seed)
    strategy = rv.OrderingStrategy.MATCH_ORDER_METIS if case["mc64"] else rv.OrderingStrategy.METIS
    solver = rv.SparseLDLT.analyze_with_matrix(s, rv.AnalyzeOptions(strategy))
    if case["form"] == "learned":
        solver.set_selector(rv.PrecisionSelector.load(
            os.path.join(os.path.dirname(rv.__file__), "data", "selector_bf16.npz")))
    opts = _options(case["form"])
    b = _rhs(s.n, case["nrhs"], seed)
    st = dict(op=case["op"], form=case["form"], host=case["host"], nrhs=case["nrhs"], solver=solver, opts=opts,
              values=s.values, b=b)
    if case["op"] == "solve" or not case["host"]:
        solver.factor(s.values, opts)  # the handle, and the factor that a solve reads
    if not case["host"]:
        st["stream"] = torch.cuda.ExternalStream(solver.stream())
        st["d_values"] = torch.from_numpy(s.values).cuda()
        st["d_scaling"] = None if solver._scaling is None else torch.from_numpy(solver._scaling).cuda()
        # columns of length n, one after another
        st["d_b"] = torch.from_numpy(np.ascontiguousarray(b.T if b.ndim == 2 else b[None, :])).cuda()
        st["d_x"] = torch.empty_like(st["d_b"])
        torch.cuda.synchronize()
    return st


def run(st):
    if st["op"] == "batch":
        x = st["batch"].factor_solve(st["values"], st["rhs"])
        return {"x": x, "inertia": [int(v) for t in st["batch"].inertias() for v in t]}
    solver, opts = st["solver"], st["opts"]
    out = {}
    if st["op"] == "step":
        if st["host"]:
            solver.factor(st["values"], opts)
        else:
            d_s = st["d_scaling"]
            solver.factor_device(st["d_values"].data_ptr(), None if d_s is None else d_s.data_ptr(), opts)
        out["inertia"] = np.array(solver.inertia())
    if st["host"]:
        out["x"] = solver.solve(st["b"]) if st["form"] == "fp64" else solver.solve_auto(st["b"])[0]
    elif st["form"] == "fp64":
        x = st["d_x"]
        with torch.cuda.stream(st["stream"]):  # the handle's stream: in order with its kernels
            x.copy_(st["d_b"])
        solver.solve_device(x.data_ptr(), st["nrhs"])
        out["x"] = x
    else:
        solver.solve_auto_device(st["d_b"].data_ptr(), st["d_x"].data_ptr())
        out["x"] = st["d_x"]
    return out


# ---- work, tolerance, reference values -----------------------------------------------------------------------


@functools.lru_cache(maxsize=64)
def _counts(matrix, g, seed):
    """(n, stored entries, entries of L, operations of the factorization) of a system's symbolic structure."""
    s = _system(matrix, g, seed)
    sym = rv.symbolic_analyze(s.n, s.colptr, s.rowidx, rv.ordering.default_order(s))
    nnz_l = flops = 0
    for b, e, r in zip(sym.sup_begin.tolist(), sym.sup_end.tolist(), np.diff(sym.pat_ptr).tolist()):
        below = np.arange(e - b - 1, -1, -1, dtype=np.float64) + r  # rows below each pivot
        nnz_l += int(below.sum()) + (e - b)
        flops += float((below * (below + 2)).sum())
    return s.n, s.rowidx.size, nnz_l, flops


def work(case):
    if case["op"] == "batch":
        systems, nrhs = _batch(case, 0)
        total = {"bytes": 0, "flops": 0.0}
        for i, (s, r) in enumerate(zip(systems, nrhs)):
            g = s.grid[0]
            n, nnz, nnz_l, fl = _counts("laplace" if i % 2 == 0 else "kkt", g, i)
            total["bytes"] += 8 * (nnz + nnz_l + 2 * n * r)
            total["flops"] += fl + 4.0 * nnz_l * r
        return total
    n, nnz, nnz_l, fl = _counts(case["matrix"], case["g"], 0)
    vectors = 16 * n * case["nrhs"]
    if case["op"] == "solve":  # the factor read once, right-hand sides in, solutions out
        return {"bytes": 8 * nnz_l + vectors, "flops": 4.0 * nnz_l * case["nrhs"]}
    return {"bytes": 8 * (nnz + nnz_l) + vectors, "flops": fl + 4.0 * nnz_l * case["nrhs"]}


def tolerance(case):
    # The backward error is near 1e-16 (1e-14 is asked of the refined forms); the condition numbers stand between
    # that and the solution.  Measured against exact(): Laplacians 2e-14 (g = 8) to 1.5e-11 (g = 80), stencils
    # 3e-12, KKT systems 3e-14 in FP64 and up to 4e-9 in the refined forms; about four times the difference of
    # two such solutions.
    if case["op"] == "batch" or case["matrix"] in ("laplace", "stencil"):
        return {"rel": 1e-10, "max": 1e-9}
    if case["form"] == "fp64":
        return {"rel": 1e-12, "max": 1e-11}
    return {"rel": 3e-8, "max": 1e-6}


def _refine(s, b, approx):
    """x of A x = b: corrections by `approx`, residuals in extended precision."""
    b2 = (b if b.ndim == 2 else b[:, None]).astype(np.longdouble)
    val = s.values.astype(np.longdouble)
    x = np.zeros_like(b2)
    starts = s.colptr[:-1]
    for _ in range(4):
        r = np.empty_like(b2)
        for j in range(b2.shape[1]):  # A is symmetric: its columns are its rows
            r[:, j] = b2[:, j] - np.add.reduceat(val * x[s.rowidx, j], starts)
        x += approx(r.astype(np.float64)).astype(np.longdouble)
    x = x.astype(np.float64)
    return x if b.ndim == 2 else x[:, 0]


def _dense_solver(s):
    a = torch.zeros(s.n, s.n, dtype=torch.float64, device="cuda")
    a[torch.from_numpy(s.rowidx).cuda(), torch.from_numpy(_csc_columns(s)).cuda()] = torch.from_numpy(s.values).cuda()
    lu, piv = torch.linalg.lu_factor(a)
    del a
    return lambda r: torch.linalg.lu_solve(lu, piv, torch.from_numpy(np.ascontiguousarray(r)).cuda()).cpu().numpy()


def _laplace_solver(s, g, seed):
    """The shifted Laplacian by its sine transform; the symmetric scaling around it is diagonal."""
    base = _laplace(g)
    sigma = base.meta["sigma"]
    d = _laplace_scaling(base, seed)[:, None]
    k = torch.arange(1, g + 1, dtype=torch.float64, device="cuda")
    h = 1.0 / (g + 1)
    q = math.sqrt(2.0 * h) * torch.sin(math.pi * h * torch.outer(k, k))
    lam = (4.0 / h ** 2) * torch.sin(0.5 * math.pi * h * k) ** 2
    den = (lam[:, None, None] + lam[None, :, None] + lam[None, None, :] - sigma)[..., None]

    def transform(t):
        for spec in ("ai,ijkr->ajkr", "bj,ajkr->abkr", "ck,abkr->abcr"):
            t = torch.einsum(spec, q, t)
        return t

    def solve(r):
        t = torch.from_numpy(r / d).cuda().reshape(g, g, g, -1)
        return transform(transform(t) / den).reshape(r.shape).cpu().numpy() / d

    return solve


def _exact_x(matrix, g, s, b, seed):
    if matrix == "laplace":
        return _refine(s, b, _laplace_solver(s, g, seed))
    if s.n > 60000:  # dense: 29 GB and a few seconds
        return None
    return _refine(s, b, _dense_solver(s))


def exact(case, seed):
    if case["op"] == "batch":
        systems, nrhs = _batch(case, seed)
        xs = []
        for i, (s, r) in enumerate(zip(systems, nrhs)):
            b = _rhs(s.n, r, seed + i)
            xs.append(_exact_x("laplace" if i % 2 == 0 else "kkt", s.grid[0], s, b, seed + i))
        return {"x": xs, "inertia": None}
    s = _system(case["matrix"], case["g"], seed)
    b = _rhs(s.n, case["nrhs"], seed)
    x = _exact_x(case["matrix"], case["g"], s, b, seed)
    if x is None:
        return None
    if not case["host"]:
        x = np.ascontiguousarray(x.T if x.ndim == 2 else x[None, :])
    out = {"x": x}
    if case["op"] == "step":
        out["inertia"] = None
    return out
