"""The SpMV variant and short-row limit a plan starts with: rows up to the limit
in the reference's order (bit-identical), those of up to 16 entries in the
order of a warp's tree (bit-identical), longer ones within the summation bound,
at the row lengths where the rules change."""
import numpy as np
import pytest

from monolish_b200 import workloads as W

pytestmark = pytest.mark.gpu


def lengths_matrix(lengths, n_cols, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n_cols, k, replace=False)) for k in lengths])
    return rp, ci.astype(np.int32), rng.uniform(-1, 1, int(rp[-1]))


def tree_sum(products):
    """A warp's xor tree over up to 32 products: l and l + 16, then l + 8, ..."""
    s = np.zeros(32, products.dtype)
    s[:len(products)] += products
    for o in (16, 8, 4, 2, 1):
        s = s[:o] + s[o:2 * o]
    return s[0]


# row lengths
CASES = {"stencil_7": [7] * 700, "up_to_8": [8, 1] * 300, "up_to_9": [9, 2] * 300,
         "all_16": [16] * 300, "0_to_17": list(range(18)) * 30, "even_33": [33] * 200,
         "one_of_33": [33] + [4] * 900, "one_of_32": [32] + [3] * 900,
         "one_of_5000": [5000] + [3] * 2000}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", sorted(CASES))
def test_defaults(handle, restatement, name, dtype):
    import torch
    from monolish_b200.device import Crs
    lengths = CASES[name]
    n_cols = 6000
    rp, ci, v = lengths_matrix(lengths, n_cols, 4)
    v = v.astype(dtype)
    n = len(lengths)
    A = Crs(handle, n, n_cols, rp, ci, v)
    assert A.tuning() == (2, 8)
    x = W.uniform_mt(n_cols, -1, 1, 2, dtype)
    y = torch.full((n,), float("nan"), device="cuda",
                   dtype=torch.float64 if dtype == np.float64 else torch.float32)
    A.matvec(torch.from_numpy(x).cuda(), y)
    got, want = y.cpu().numpy(), restatement.spmv(rp, ci, v, x)
    lens = np.diff(rp)
    assert np.array_equal(got[lens <= 8], want[lens <= 8])
    for i in np.nonzero((lens > 8) & (lens <= 32))[0]:
        e = slice(rp[i], rp[i + 1])
        assert got[i] == tree_sum(v[e] * x[ci[e]])
    scale = restatement.spmv(rp, ci, np.abs(v), np.abs(x))
    eps = np.finfo(dtype).eps
    assert np.all(np.abs(got - want) <= 4 * lens * eps * scale)
    A.close()
