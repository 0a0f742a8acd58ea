"""COO sorting and CRS transposition by grouping, where it changes form: rows
around the warp's segment and the CTA's limit, rows past it (the radix sort),
far more rows than entries (the radix sort), empty rows, equal entries across
segments.  Orders, indices and values are bit-exact against the restatement.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEG, LONG = 384, 16384  # group sizes of the warp and the CTA kernel


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _coo(lengths, n_cols, seed, dtype, distinct):
    """Rows of the given lengths in shuffled order; columns repeat when fewer
    than `distinct` are drawn from."""
    rng = np.random.default_rng(seed)
    row = np.repeat(np.arange(len(lengths)), lengths).astype(np.int32)
    col = rng.integers(0, min(n_cols, distinct), len(row)).astype(np.int32)
    p = rng.permutation(len(row))
    return row[p], col[p], rng.uniform(-1, 1, len(row)).astype(dtype)


LENGTHS = {"stencil_33_rows": [7] * 33,
           "segment_edges": [SEG - 1, 1, SEG, 0, SEG + 1, 3, 0, 0, 2 * SEG],
           "segments_of_200": [200] * 65,
           "one_row": [1025],
           "cta_edges": [5, 1023, 1024, 1025, LONG, LONG - 1, 2],
           "past_the_cta": [5, LONG + 1, 7],
           "many_empty_rows": [3] + [0] * 40000 + [2]}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("merge", [True, False])
@pytest.mark.parametrize("distinct", [50, 1 << 30])
@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_coo_sort_group_sizes(handle, restatement, name, distinct, merge, dtype):
    from monolish_b200 import device as D
    lengths, n_cols = LENGTHS[name], 100000
    row, col, val = _coo(lengths, n_cols, 11, dtype, distinct)
    dr, dc, dv = _dev(row), _dev(col), _dev(val)
    cnt = D.coo_sort(handle, len(lengths), n_cols, dr, dc, dv, merge=merge)
    er, ec, ev = restatement.coo_sort(row, col, val.astype(np.float64), merge)
    assert cnt == len(er)
    assert np.array_equal(dr.cpu().numpy()[:cnt], er)
    assert np.array_equal(dc.cpu().numpy()[:cnt], ec)
    assert np.array_equal(dv.cpu().numpy()[:cnt], ev.astype(dtype))
    rp = D.coo_to_csr(handle, len(lengths), dr, cnt).cpu().numpy()
    assert np.array_equal(rp, restatement.coo_rowptr(len(lengths), er))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_transpose_group_sizes(handle, restatement, name, dtype):
    """The lengths are column lengths here: a CRS whose columns are that long."""
    from monolish_b200 import device as D
    lengths = LENGTHS[name]
    n_rows = max(max(lengths), 1)
    rng = np.random.default_rng(12)
    row = np.concatenate([rng.choice(n_rows, k, replace=False) for k in lengths])
    col = np.repeat(np.arange(len(lengths)), lengths)
    o = np.lexsort((col, row))
    row, ci = row[o], col[o].astype(np.int32)
    rp = np.searchsorted(row, np.arange(n_rows + 1)).astype(np.int32)
    v = rng.uniform(-1, 1, len(ci)).astype(dtype)
    rp_t, ci_t, v_t = D.csr_transpose(handle, n_rows, len(lengths), _dev(rp), _dev(ci), _dev(v))
    e_rp, e_ci, e_v = restatement.csr_transpose(rp, ci, v.astype(np.float64), len(lengths))
    assert np.array_equal(rp_t.cpu().numpy(), e_rp)
    assert np.array_equal(ci_t.cpu().numpy(), e_ci)
    assert np.array_equal(v_t.cpu().numpy(), e_v.astype(dtype))


def test_sort_between_solves(handle):
    """Sorting uses the handle's work buffer: a solve before and after it, on
    the same handle, gives the same bits."""
    import torch
    from monolish_b200 import _abi
    from monolish_b200 import device as D
    from monolish_b200 import workloads as W
    n, rp, ci, v = W.poisson3d(20)
    A = D.Crs(handle, n, n, rp, ci, v)
    b = torch.ones(n, dtype=torch.float64, device="cuda")

    def solve():
        x = torch.zeros_like(b)
        D.cg_solve(A, b, x, 1e-8, 1000, engine=_abi.ENGINE_KERNELS)
        return x
    x1 = solve()
    row, col, val = _coo([40] * 20000, 5000, 3, np.float64, 1 << 30)
    D.coo_sort(handle, 20000, 5000, _dev(row), _dev(col), _dev(val))
    assert torch.equal(x1, solve())
    A.close()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n_rows", [300, 65537, 4000000])
@pytest.mark.parametrize("k,order", [((1 << 22) - 1, "shuffled"), ((1 << 22) + 777, "shuffled"),
                                     ((1 << 22) + 777, "rows")])
def test_two_scatters(handle, n_rows, k, order, dtype):
    """Entries in no order, just below and above the size from which they go to
    ranges of rows first, and in row order (one scatter); against numpy."""
    from monolish_b200 import device as D
    rng = np.random.default_rng(k + n_rows)
    row = rng.integers(0, n_rows, k, dtype=np.int32)
    if order == "rows":
        row.sort()
    # few columns in long rows, so that entries repeat
    col = rng.integers(0, 3 if n_rows > 1000 else 20000, k, dtype=np.int32)
    val = rng.uniform(-1, 1, k).astype(dtype)
    o = np.lexsort((np.arange(k), col, row))
    last = np.ones(k, bool)
    last[:-1] = (row[o][1:] != row[o][:-1]) | (col[o][1:] != col[o][:-1])
    dr, dc, dv = _dev(row), _dev(col), _dev(val)
    cnt = D.coo_sort(handle, n_rows, 20000, dr, dc, dv, merge=True)
    assert cnt == int(last.sum())
    assert np.array_equal(dr.cpu().numpy()[:cnt], row[o][last])
    assert np.array_equal(dc.cpu().numpy()[:cnt], col[o][last])
    assert np.array_equal(dv.cpu().numpy()[:cnt], val[o][last])


@pytest.mark.parametrize("row", [[0, 2, 1, 3], [0, 1, 5, 5], [-1, 0, 1, 2]])
def test_refused_rows_leave_the_output(handle, row):
    """Rows out of order or out of range: the error, and row_ptr as it was."""
    import torch
    from monolish_b200 import _abi
    from monolish_b200.device import ptr
    d_row = _dev(np.array(row, np.int32))
    rp = torch.full((6,), 77, dtype=torch.int32, device="cuda")
    st = handle.lib.mlsh_coo_to_csr(handle.h, 5, 4, ptr(d_row), ptr(rp))
    assert st == _abi.ERR_INVALID_CSR
    assert (rp == 77).all()
