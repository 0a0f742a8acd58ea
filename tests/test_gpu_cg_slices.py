"""CG in slice form where it changes shape: rows per CTA around the thread
count and the slices' 32 rows, matrices that stay in shared memory, that
partly do and that are streamed, one cluster and the whole GPU, rows up to and
past the form's 16 entries, and both precisions.

Against the restatement's CG (the reference's recurrence): same status,
iterations within +-2 % (at least one); the true residual near the tolerance
and the solution within what it leaves."""
import numpy as np
import pytest

from monolish_b200 import _abi
from monolish_b200 import workloads as W

pytestmark = pytest.mark.gpu


def shifted(rp, ci, v, shift):
    """A + shift I: few iterations, so that large cases stay quick."""
    v = v.copy()
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    v[rows == ci] += shift
    return rp, ci, v


def banded(n, width, seed):
    """Symmetric, diagonally dominant, rows of up to 2 width + 1 entries with
    some missing (uneven rows)."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), width)
    j = i + np.tile(np.arange(1, width + 1) * 7, n)
    keep = (j < n) & (rng.random(len(i)) < 0.9)
    keep |= (i % 97 == 0) & (j < n)
    i, j = i[keep], j[keep]
    w = rng.uniform(-1, 1, len(i))
    row, col = np.concatenate([i, j, np.arange(n)]), np.concatenate([j, i, np.arange(n)])
    val = np.concatenate([w, w, np.zeros(n)])
    o = np.lexsort((col, row))
    row, col, val = row[o], col[o], val[o]
    rp = np.searchsorted(row, np.arange(n + 1)).astype(np.int32)
    diag = row == col
    val[diag] = np.bincount(row, np.abs(val), n) + 1.0
    return rp, col.astype(np.int32), val


def check(handle, restatement, mat, dtype=np.float64, precond=_abi.PRECOND_JACOBI,
          engine=_abi.ENGINE_AUTO, rows=0, x0=False, tol=None):
    import torch
    from monolish_b200 import device as D
    rp, ci, v = mat
    n = len(rp) - 1
    v = v.astype(dtype)
    xt = W.uniform_mt(n, -1, 1, 0, dtype)
    b = restatement.spmv(rp, ci, v, xt)
    tol = (1e-10 if dtype == np.float64 else 1e-5) * float(np.linalg.norm(b.astype(np.float64)))
    start = W.uniform_mt(n, -1, 1, 5, dtype) if x0 else np.zeros(n, dtype)
    A = D.Crs(handle, n, n, rp, ci, v)
    x = torch.from_numpy(start.copy()).cuda()
    hist = np.zeros(5)
    r = D.cg_solve(A, torch.from_numpy(b).cuda(), x, tol, 5000, precond=precond, engine=engine,
                   cluster_rows=rows, history=hist)
    st, it, _, want = restatement.cg(rp, ci, v, b, start, tol, 5000, precond=precond)
    A.close()
    assert r.status == st == 0
    assert abs(r.iters - it) <= max(1, it // 50), (r.iters, it)
    assert (hist[:min(5, r.iters)] >= 0).all() and (r.iters > 5 or hist[r.iters - 1] == r.resid)
    assert r.iters <= 5 or (hist > 0).all()
    # the true residual (FP32: the recursive one drifts from it by some units
    # in the last place of b), and with lambda_min >= 1/2 what it leaves in x
    got = x.cpu().numpy().astype(np.float64)
    rows_of = np.repeat(np.arange(n), np.diff(rp))
    res = b - np.bincount(rows_of, v.astype(np.float64) * got[ci], n)
    left = float(np.linalg.norm(res))
    assert left < (2 * tol if dtype == np.float64 else 6 * tol), (left, tol)
    assert np.abs(got - xt).max() <= 2 * left + (1e-12 if dtype == np.float64 else 1e-5)


# rows: one CTA and its edges, cluster slices of 1,024 .. 8,192 rows with a last
# CTA of one row and of all, and the same systems on the whole GPU
@pytest.mark.parametrize("engine", [_abi.ENGINE_AUTO, _abi.ENGINE_GRID])
@pytest.mark.parametrize("n", [1, 31, 33, 1023, 1025, 16384, 16385, 32768, 32769, 65536, 65537])
def test_sizes(handle, restatement, n, engine):
    nx = max(1, int(np.sqrt(n)))
    while n % nx:
        nx -= 1
    check(handle, restatement, shifted(*W.poisson2d(nx, n // nx)[1:], 0.5), engine=engine)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("rows", [1024, 2048, 4096, 8192, 16384])
def test_rows_per_cta(handle, restatement, rows, dtype):
    """Resident, partly resident and streamed matrices on one cluster."""
    if dtype == np.float64 and rows == 16384:
        pytest.skip("8,192 rows a CTA at most in FP64")
    check(handle, restatement, shifted(*W.poisson2d(121, 119)[1:], 0.5), dtype,
          engine=_abi.ENGINE_CLUSTER, rows=rows)


@pytest.mark.parametrize("m", [33, 64, 84, 85])  # 84^3: 4,005 rows a CTA; 85^3: past them
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_whole_gpu_3d(handle, restatement, m, dtype):
    check(handle, restatement, shifted(*W.vardiff3d(m, m, m, 3, 0)[1:], 0.7), dtype,
          engine=_abi.ENGINE_GRID)


@pytest.mark.parametrize("n,engine", [(2500, _abi.ENGINE_AUTO), (70000, _abi.ENGINE_AUTO),
                                      (70000, _abi.ENGINE_GRID)])
@pytest.mark.parametrize("width", [1, 4, 7, 8])
def test_row_lengths(handle, restatement, n, engine, width):
    """Rows of up to 3, 9, 15 and 17 entries (the last past the slice form)."""
    check(handle, restatement, banded(n, width, width), engine=engine)


@pytest.mark.parametrize("n,engine", [(900, _abi.ENGINE_AUTO), (72900, _abi.ENGINE_AUTO),
                                      (72900, _abi.ENGINE_GRID)])
def test_no_preconditioner_and_initial_guess(handle, restatement, n, engine):
    m = int(np.sqrt(n))
    check(handle, restatement, shifted(*W.poisson2d(m, m)[1:], 0.5),
          precond=_abi.PRECOND_NONE, engine=engine, x0=True)


def test_whole_gpu_stops(handle):
    """maxiter, a budget that runs out, NaN, then a solve on the same handle;
    a repeat gives the same bits."""
    import torch
    from monolish_b200 import device as D
    n, rp, ci, v = W.poisson2d(310, 300)
    A = D.Crs(handle, n, n, rp, ci, v)
    b = torch.ones(n, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    grid = dict(engine=_abi.ENGINE_GRID)
    r = D.cg_solve(A, b, x, 0.0, 7, **grid)
    assert (r.status, r.iters) == (_abi.SOLVER_MAXITER, 7)
    with pytest.raises(_abi.MlshError) as e:
        D.cg_solve(A, b, x.zero_(), 1e-8, 100000, time_limit=1e-7, **grid)
    assert e.value.status == _abi.ERR_TIMEOUT
    bad = b.clone()
    bad[5] = float("nan")
    assert D.cg_solve(A, bad, x.zero_(), 1e-8, 1000, **grid).status == _abi.SOLVER_RESIDUAL_NAN
    x1, x2 = torch.zeros_like(b), torch.zeros_like(b)
    r1 = D.cg_solve(A, b, x1, 1e-8, 100000, **grid)
    r2 = D.cg_solve(A, b, x2, 1e-8, 100000, **grid)
    assert r1.status == 0 and r1.iters == r2.iters and torch.equal(x1, x2)
    A.close()


def test_same_bits_beside_a_server(handle):
    """Which kernels solve a system does not depend on what else the process
    has: an open server changes no bit."""
    import torch
    from monolish_b200 import device as D
    n, rp, ci, v = W.poisson2d(310, 300)
    A = D.Crs(handle, n, n, rp, ci, v)
    b = torch.ones(n, dtype=torch.float64, device="cuda")
    x1, x2 = torch.zeros_like(b), torch.zeros_like(b)
    r1 = D.cg_solve(A, b, x1, 1e-8, 100000)
    s = D.Server(memory_budget=1 << 28, n_lanes=1)
    r2 = D.cg_solve(A, b, x2, 1e-8, 100000)
    s.close()
    assert r1.status == 0 and r1.iters == r2.iters and torch.equal(x1, x2)
    A.close()


def test_batch_of_many_shapes(handle, restatement):
    """One batch over all slice widths, a system past the slice form in it."""
    import torch
    from monolish_b200 import device as D
    mats = [shifted(*W.poisson2d(a, b)[1:], 0.5)
            for a, b in ((1, 1), (5, 7), (40, 26), (64, 33), (100, 82), (99, 90), (160, 110))]
    mats.append(banded(3000, 9, 1))
    B = D.Batch(handle, mats)
    bs, xts = [], []
    for k, (rp, ci, v) in enumerate(mats):
        xt = W.uniform_mt(len(rp) - 1, -1, 1, k)
        xts.append(xt)
        bs.append(restatement.spmv(rp, ci, v, xt))
    tol = np.array([1e-10 * np.linalg.norm(b) for b in bs])
    db = torch.from_numpy(np.concatenate(bs)).cuda()
    dx = torch.zeros_like(db)
    status, iters, _ = B.solve("cg", db, dx, tol, 5000)
    assert (status == 0).all()
    for k, x in enumerate(np.split(dx.cpu().numpy(), np.cumsum([len(b) for b in bs])[:-1])):
        rp, ci, v = mats[k]
        _, it, _, _ = restatement.cg(rp, ci, v, bs[k], np.zeros(len(x)), tol[k], 5000)
        assert abs(iters[k] - it) <= max(1, it // 50)
        assert np.abs(x - xts[k]).max() < 1e-8
    B.close()
