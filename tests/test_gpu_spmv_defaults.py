"""The SpMV variant and short-row limit a plan starts with: rows up to the limit
in the reference's order (bit-identical), longer ones within the summation
bound, at the row lengths and the unevenness where the rule changes."""
import numpy as np
import pytest

from monolish_b200 import workloads as W

pytestmark = pytest.mark.gpu


def lengths_matrix(lengths, n_cols, seed):
    rng = np.random.default_rng(seed)
    rp = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(n_cols, k, replace=False)) for k in lengths])
    return rp, ci.astype(np.int32), rng.uniform(-1, 1, int(rp[-1]))


# (row lengths, the limit to expect, uneven)
CASES = {"stencil_7": ([7] * 700, 8, False), "up_to_8": ([8, 1] * 300, 8, False),
         "up_to_9": ([9, 2] * 300, 16, False), "all_16": ([16] * 300, 16, False),
         "up_to_17": ([17, 3] * 300, 16, False), "even_33": ([33] * 200, 16, False),
         "one_of_33": ([33] + [4] * 900, 16, True), "one_of_32": ([32] + [3] * 900, 16, False),
         "one_of_5000": ([5000] + [3] * 2000, 16, True)}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", sorted(CASES))
def test_defaults(handle, restatement, name, dtype):
    import torch
    from monolish_b200.device import Crs
    lengths, limit, uneven = CASES[name]
    n_cols = 6000
    rp, ci, v = lengths_matrix(lengths, n_cols, 4)
    v = v.astype(dtype)
    n = len(lengths)
    A = Crs(handle, n, n_cols, rp, ci, v)
    variant, short = A.tuning()
    assert short == limit
    assert variant == (0 if uneven and dtype == np.float64 else 2)
    x = W.uniform_mt(n_cols, -1, 1, 2, dtype)
    y = torch.full((n,), float("nan"), device="cuda",
                   dtype=torch.float64 if dtype == np.float64 else torch.float32)
    A.matvec(torch.from_numpy(x).cuda(), y)
    got, want = y.cpu().numpy(), restatement.spmv(rp, ci, v, x)
    lens = np.diff(rp)
    assert np.array_equal(got[lens <= limit], want[lens <= limit])
    scale = restatement.spmv(rp, ci, np.abs(v), np.abs(x))
    eps = np.finfo(dtype).eps
    assert np.all(np.abs(got - want) <= 4 * lens * eps * scale)
    A.close()
