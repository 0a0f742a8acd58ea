"""The calls this library is timed on, through its public entry points.

A program that uses the library does four things with it: it assembles a CRS
matrix from triplets, it multiplies with it, it runs Krylov solves on it (one
system at a time, or many small ones together), and it writes its own steps
with the vector BLAS.  The listed cases are those calls at the sizes of the
repository's own workloads and tests, small and large, FP64 / FP32 / mixed;
``draw`` gives more of the same ranges, odd sizes among them.

What a program keeps between calls (matrix, plan, preconditioner, batch) is
made in ``prepare``; ``run`` is one pass of the call itself.
"""
import math

import numpy as np
import torch

from monolish_b200 import _abi
from monolish_b200 import device as D
from monolish_b200 import workloads as W


def listed():
    return [
        # a user's own solver step on a small grid: seven BLAS calls, each a
        # few microseconds, two of them waited for (blas::dot returns a value)
        {"name": "blas_step_poisson2d_127x129_f64", "kind": "blas", "grid": 127,
         "grid2": 129, "dtype": "f64"},
        # blas::matvec, the stencil matrix of the default benchmark
        {"name": "spmv_poisson3d_256_f64", "kind": "spmv", "matrix": "poisson3d", "size": 256,
         "dtype": "f64", "transpose": False},
        # single precision, an odd grid (rows of x and y not 16-byte multiples)
        {"name": "spmv_poisson3d_201_f32", "kind": "spmv", "matrix": "poisson3d", "size": 201,
         "dtype": "f32", "transpose": False},
        # rows of very uneven length with random columns (a graph's matrix)
        {"name": "spmv_zipf_4194304_f64", "kind": "spmv", "matrix": "zipf", "size": 4194304,
         "dtype": "f64", "transpose": False},
        # blas::matvec_T of such a matrix, single precision, odd size
        {"name": "spmv_t_zipf_1000003_f32", "kind": "spmv", "matrix": "zipf", "size": 1000003,
         "dtype": "f32", "transpose": True},
        # a small system solved alone: the latency of one iteration counts
        {"name": "cg_poisson2d_128_f64", "kind": "solve", "method": "cg", "matrix": "poisson2d",
         "size": 128, "precision": "f64"},
        # a million rows, variable coefficients, odd grid
        {"name": "cg_vardiff3d_101_f64", "kind": "solve", "method": "cg", "matrix": "vardiff3d",
         "size": 101, "precision": "f64"},
        # a large nonsymmetric system, in double and in mixed precision
        {"name": "bicgstab_convdiff_160_f64", "kind": "solve", "method": "bicgstab",
         "matrix": "convdiff3d", "size": 160, "precision": "f64"},
        {"name": "bicgstab_convdiff_160_mixed", "kind": "solve", "method": "bicgstab",
         "matrix": "convdiff3d", "size": 160, "precision": "mixed"},
        # a sweep preconditioner (equation::IC) in CG
        {"name": "ic_cg_poisson3d_49_f64", "kind": "precond", "precond": "ic",
         "matrix": "poisson3d", "size": 49},
        # many uneven independent systems in one call
        {"name": "batch_cg_256_f64", "kind": "batch", "count": 256, "lo": 1000, "hi": 100000,
         "precision": "f64"},
        # triplets in any order, some of them repeated, to a CRS matrix
        {"name": "assemble_poisson3d_128_f64", "kind": "assemble", "grid": 128, "extra": 0.1,
         "order": "shuffled", "dtype": "f64"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["blas", "spmv", "spmv", "solve", "solve", "precond", "batch", "assemble"])
    if kind == "blas":
        return {"kind": kind, "grid": _log_int(rng, 24, 1200), "grid2": _log_int(rng, 24, 1200),
                "dtype": rng.choice(["f64", "f32"])}
    if kind == "spmv":
        matrix = rng.choice(["poisson2d", "poisson3d", "convdiff3d", "zipf"])
        lo, hi = {"poisson2d": (40, 3000), "poisson3d": (16, 250), "convdiff3d": (16, 200),
                  "zipf": (5000, 4000000)}[matrix]
        return {"kind": kind, "matrix": matrix, "size": _log_int(rng, lo, hi),
                "dtype": rng.choice(["f64", "f32"]), "transpose": rng.random() < 0.25}
    if kind == "solve":
        method = rng.choice(["cg", "cg", "bicgstab"])
        if method == "cg":
            matrix = rng.choice(["poisson2d", "vardiff3d"])
            size = _log_int(rng, 32, 320) if matrix == "poisson2d" else _log_int(rng, 12, 120)
        else:
            matrix, size = "convdiff3d", _log_int(rng, 12, 150)
        return {"kind": kind, "method": method, "matrix": matrix, "size": size,
                "precision": rng.choice(["f64", "mixed"])}
    if kind == "precond":
        precond = rng.choice(["ic", "ilu", "sor"])
        if precond == "sor":
            return {"kind": kind, "precond": precond, "matrix": "poisson2d",
                    "size": _log_int(rng, 32, 128)}
        return {"kind": kind, "precond": precond,
                "matrix": "poisson3d" if precond == "ic" else "convdiff3d",
                "size": rng.choice([64, 96]) if rng.random() < 0.3 else _log_int(rng, 16, 48)}
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 16, 250), "lo": 1000,
                "hi": _log_int(rng, 3000, 90000), "precision": rng.choice(["f64", "mixed"])}
    return {"kind": kind, "grid": _log_int(rng, 16, 125), "extra": rng.choice([0.0, 0.1, 0.5]),
            "order": rng.choice(["shuffled", "rows"]), "dtype": rng.choice(["f64", "f32"])}


# ------------------------------------------------------------------ inputs --
def _np_dtype(name):
    return np.float32 if name == "f32" else np.float64


def _matrix(case, seed):
    """(n, row_ptr, col_ind, val) on the host; the random families from the seed."""
    m, s = case["matrix"], case["size"]
    if m == "poisson2d":
        return W.poisson2d(s)
    if m == "poisson3d":
        return W.poisson3d(s)
    if m == "convdiff3d":
        return W.convdiff3d(s)
    if m == "vardiff3d":
        return W.vardiff3d(s, s, s, seed, 0)
    return W.zipf(s, seed=seed + 1)


def _uniform(n, seed, dtype=torch.float64):
    """n values of U[-1, 1] on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(n, generator=g, device="cuda", dtype=dtype) * 2 - 1


def _product(n, rp, ci, v, x):
    """A x in 64 bits by plain torch (sums along the rows of A)."""
    lengths = torch.from_numpy(np.diff(rp)).cuda().long()
    cols = torch.from_numpy(np.ascontiguousarray(ci)).cuda().long()
    prod = torch.from_numpy(np.ascontiguousarray(v)).cuda().double() * x.double()[cols]
    return torch.segment_reduce(prod, "sum", lengths=lengths, initial=0.0)


def _tol(case):
    """Relative residual the solves go to (the repository's own settings)."""
    return 1e-8 if case["kind"] == "batch" else 1e-10


def _triplets(case, seed):
    """(n, row, col, val) on the GPU: a 7-point matrix's entries, a share of
    them given again with another value, in random or in row order."""
    n, rp, ci, _ = W.poisson3d(case["grid"])
    lengths = torch.from_numpy(np.diff(rp)).cuda().long()
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), lengths)
    col = torch.from_numpy(ci).cuda().long()
    g = torch.Generator(device="cuda").manual_seed(seed)
    extra = int(case["extra"] * row.numel())
    if extra:
        again = torch.randint(0, row.numel(), (extra,), generator=g, device="cuda")
        row, col = torch.cat([row, row[again]]), torch.cat([col, col[again]])
    if case["order"] == "shuffled":
        perm = torch.randperm(row.numel(), generator=g, device="cuda")
        row, col = row[perm], col[perm]
    else:
        # a row's entries together (its columns in the order they were given)
        row, perm = torch.sort(row, stable=True)
        col = col[perm]
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    val = torch.rand(row.numel(), generator=g, device="cuda", dtype=dt) * 2 - 1
    return n, row.int(), col.int(), val


def _batch_systems(case, seed):
    """Variable-coefficient diffusion systems: the case's sizes, the seed's values."""
    systems = []
    for k, n in enumerate(W.loguniform_sizes(case["count"], case["lo"], case["hi"], 3)):
        nx, ny = W.grid2d_for(int(n))
        systems.append(W.vardiff2d(nx, ny, seed, k)[1:])
    return systems


def _batch_solution(case, seed, total):
    return _uniform(total, seed)


def prepare(case, seed):
    kind = case["kind"]
    h = D.Handle()
    st = {"case": case, "h": h}
    if kind == "assemble":
        n, row, col, val = _triplets(case, seed)
        st.update(n=n, src=(row, col, val),
                  buf=(torch.empty_like(row), torch.empty_like(col), torch.empty_like(val)))
        return st
    if kind == "batch":
        systems = _batch_systems(case, seed)
        B = D.Batch(h, systems)
        total = int(B.row_off[-1])
        x = _batch_solution(case, seed, total)
        b = torch.empty_like(x)
        tol = np.empty(len(systems))
        for k, (rp, ci, v) in enumerate(systems):
            lo, hi = int(B.row_off[k]), int(B.row_off[k + 1])
            b[lo:hi] = _product(hi - lo, rp, ci, v, x[lo:hi])
            tol[k] = _tol(case) * float(torch.linalg.vector_norm(b[lo:hi]))
        st.update(B=B, b=b, tol=tol, x=torch.zeros_like(x))
        return st
    if kind == "blas":
        n, rp, ci, v = W.poisson2d(case["grid"], case["grid2"])
        dt = _np_dtype(case["dtype"])
        tdt = torch.float32 if dt == np.float32 else torch.float64
        st.update(A=D.Crs(h, n, n, rp, ci, v.astype(dt)), x0=_uniform(n, seed, tdt),
                  r0=_uniform(n, seed + 1, tdt))
        st.update({k: torch.empty_like(st["x0"]) for k in ("x", "r", "q")})
        return st
    n, rp, ci, v = _matrix(case, seed)
    if kind == "spmv":
        dt = _np_dtype(case["dtype"])
        tdt = torch.float32 if dt == np.float32 else torch.float64
        st.update(A=D.Crs(h, n, n, rp, ci, v.astype(dt)), x=_uniform(n, seed, tdt),
                  y=torch.empty(n, dtype=tdt, device="cuda"))
        return st
    x = _uniform(n, seed)
    b = _product(n, rp, ci, v, x)
    st.update(A=D.Crs(h, n, n, rp, ci, v), b=b, x=torch.zeros_like(b),
              tol=_tol(case) * float(torch.linalg.vector_norm(b)))
    if kind == "precond":
        code = {"ic": _abi.PRECOND_IC, "ilu": _abi.PRECOND_ILU, "sor": _abi.PRECOND_SOR}
        st["pc"] = D.Precond(st["A"], code[case["precond"]])
    return st


# ----------------------------------------------------------------- one pass --
def run(state):
    case, h = state["case"], state["h"]
    kind = case["kind"]
    if kind == "blas":
        A, x, r, q = state["A"], state["x"], state["r"], state["q"]
        h.copy(state["x0"], x)
        h.copy(state["r0"], r)
        A.matvec(r, q)
        alpha = h.dot(r, r) / h.dot(r, q)
        h.axpy(alpha, r, x)
        h.axpy(-alpha, q, r)
        return {"x": x, "r": r, "norm": h.nrm2(r)}
    if kind == "spmv":
        (state["A"].matvec_t if case["transpose"] else state["A"].matvec)(state["x"], state["y"])
        return state["y"]
    if kind == "assemble":
        row, col, val = state["buf"]
        for dst, src in zip(state["buf"], state["src"]):
            dst.copy_(src)
        k = D.coo_sort(h, state["n"], state["n"], row, col, val, merge=True)
        rp = D.coo_to_csr(h, state["n"], row, k)
        return {"row_ptr": rp, "col": col[:k], "val": val[:k]}
    x = state["x"]
    x.zero_()
    if kind == "batch":
        B = state["B"]
        if case["precision"] == "mixed":
            B.solve_mixed(state["b"], x, state["tol"], 100000)
        else:
            B.solve("cg", state["b"], x, state["tol"], 100000)
        return x
    A, b, tol = state["A"], state["b"], state["tol"]
    if kind == "precond":
        solve = D.bicgstab_solve_precond if case["precond"] == "ilu" else D.cg_solve_precond
        solve(A, state["pc"], b, x, tol, 100000)
    elif case["precision"] == "mixed":
        (D.cg_solve_mixed if case["method"] == "cg" else D.bicgstab_solve_mixed)(A, b, x, tol,
                                                                                 100000)
    else:
        (D.cg_solve if case["method"] == "cg" else D.bicgstab_solve)(A, b, x, tol, 100000)
    return x


# ---------------------------------------------------------- work, tolerance --
def _counts(case):
    """(rows, nonzeros) of one case, without making it (random ones: expected)."""
    if case["kind"] == "batch":
        lo, hi = case["lo"], case["hi"]
        n = case["count"] * (hi - lo) / math.log(hi / lo)
        return n, 5 * n
    if case["kind"] == "blas":
        a, b = case["grid"], case["grid2"]
        return a * b, 5 * a * b - 2 * (a + b)
    if case["kind"] == "assemble":
        m, s = "poisson3d", case["grid"]
    else:
        m, s = case["matrix"], case["size"]
    if m == "poisson2d":
        return s * s, 5 * s * s - 4 * s
    if m == "zipf":
        # mean of Zipf(2) lengths cut at 10,000: H(10000) / H2(10000)
        return s, 5.95 * s
    return s ** 3, 7 * s ** 3 - 6 * s * s


def _iterations(case):
    """About how many iterations a solve takes (only its scale matters here)."""
    if case["kind"] == "batch":
        return 3.0 * math.sqrt(case["hi"]) / 2
    s = case["size"]
    if case["kind"] == "precond":
        return {"ic": 1.1, "ilu": 0.12, "sor": 1.7}[case["precond"]] * s
    return {"poisson2d": 3.0, "vardiff3d": 6.0, "convdiff3d": 1.7}[case["matrix"]] * s


def work(case):
    """Bytes: each input read and each output written once.  Operations: two a
    stored entry a product, and the vector updates of the iterations."""
    n, nnz = _counts(case)
    kind = case["kind"]
    V = 4 if case.get("dtype") == "f32" else 8
    matrix = nnz * (V + 4) + (n + 1) * 4
    if kind == "spmv":
        return {"bytes": matrix + 2 * n * V, "flops": 2 * nnz}
    if kind == "blas":
        return {"bytes": matrix + 4 * n * V, "flops": 2 * nnz + 10 * n}
    if kind == "assemble":
        given = nnz * (1 + case["extra"])
        return {"bytes": given * (V + 8) + nnz * (V + 4) + (n + 1) * 4, "flops": 0}
    two = case.get("method") == "bicgstab" or case.get("precond") == "ilu"
    per = (4 * nnz + 22 * n) if two else (2 * nnz + 11 * n)
    if kind == "precond":
        per += (2 if two else 1) * 2 * nnz
    return {"bytes": matrix + 2 * n * V, "flops": per * _iterations(case)}


def tolerance(case):
    kind = case["kind"]
    if kind == "assemble":
        return "exact"
    if kind in ("spmv", "blas"):
        return {"rel": 4e-7} if case["dtype"] == "f32" else {"rel": 2e-15, "max": 1e-12}
    # a solve stops at a relative residual: two correct ones differ by what
    # that leaves in x, which grows with the matrix's condition
    return {"rel": 1e-4 if kind == "batch" else 3e-7, "max": 1e-3 if kind == "batch" else 1e-5}


def exact(case, seed):
    kind = case["kind"]
    if kind == "assemble":
        n, row, col, val = _triplets(case, seed)
        key = row.long() * n + col.long()
        key, perm = torch.sort(key, stable=True)
        last = torch.ones_like(key, dtype=torch.bool)
        last[:-1] = key[1:] != key[:-1]
        rows = key[last] // n
        rp = torch.searchsorted(rows, torch.arange(n + 1, device="cuda")).int()
        return {"row_ptr": rp, "col": (key[last] % n).int(), "val": val[perm][last].double()}
    if kind == "batch":
        total = sum(len(rp) - 1 for rp, _, _ in _batch_systems(case, seed))
        return _batch_solution(case, seed, total)
    if kind == "blas":
        n, rp, ci, v = W.poisson2d(case["grid"], case["grid2"])
        tdt = torch.float32 if case["dtype"] == "f32" else torch.float64
        x, r = _uniform(n, seed, tdt).double(), _uniform(n, seed + 1, tdt).double()
        q = _product(n, rp, ci, v, r)
        alpha = torch.dot(r, r) / torch.dot(r, q)
        x, r = x + alpha * r, r - alpha * q
        return {"x": x, "r": r, "norm": float(torch.linalg.vector_norm(r))}
    n, rp, ci, v = _matrix(case, seed)
    if kind == "spmv":
        dt = _np_dtype(case["dtype"])
        x = _uniform(n, seed, torch.float32 if dt == np.float32 else torch.float64).double()
        v = v.astype(dt)
        if not case["transpose"]:
            return _product(n, rp, ci, v, x)
        lengths = torch.from_numpy(np.diff(rp)).cuda().long()
        prod = torch.from_numpy(v).cuda().double() * torch.repeat_interleave(x, lengths)
        out = torch.zeros(n, dtype=torch.float64, device="cuda")
        return out.index_add_(0, torch.from_numpy(ci).cuda().long(), prod)
    # b was made as A x: the solution is that x
    return _uniform(n, seed)
