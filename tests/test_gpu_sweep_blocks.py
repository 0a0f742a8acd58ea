"""Row blocks of the sweeps on grids whose lines are not multiples of 32 rows.

Blocks end at 32 rows and, where that shortens the dependency chain, at rows
that do not depend on their predecessor.  Lines just below, at and above a
block's 32 rows and twice that, lines of a few rows (where the plain blocks
stay), and a matrix with no line structure; systems in the single-CTA, the
cluster and the flag-synchronized sweeps, each asserted to run in its form.  Factors bit-identical to the sequential
restatement, applies within the sweeps' bars (1e-12 FP64 / 1e-5 FP32).
"""
import numpy as np
import pytest

from monolish_b200 import _abi
from monolish_b200 import workloads as W

pytestmark = pytest.mark.gpu

SOR, IC, ILU = _abi.PRECOND_SOR, _abi.PRECOND_IC, _abi.PRECOND_ILU


def permuted(rp, ci, v, seed):
    """P A P^T for a random P: no line structure left."""
    n = len(rp) - 1
    p = np.random.default_rng(seed).permutation(n)
    inv = np.argsort(p)
    rows = []
    for i in range(n):
        j = p[i]
        c, w = inv[ci[rp[j]:rp[j + 1]]], v[rp[j]:rp[j + 1]]
        o = np.argsort(c)
        rows.append((c[o], w[o]))
    return (np.concatenate([[0], np.cumsum([len(c) for c, _ in rows])]).astype(np.int32),
            np.concatenate([c for c, _ in rows]).astype(np.int32),
            np.concatenate([w for _, w in rows]))


def banded(n, offsets, line):
    """Symmetric, diagonally dominant: entries at +-offsets; the offset 1 stops
    at the ends of lines."""
    rng = np.random.default_rng(len(offsets))
    row, col, val = [np.arange(n)], [np.arange(n)], [np.full(n, 2.0 * len(offsets) + 1)]
    for o in offsets:
        i = np.arange(n - o)
        if o == 1:
            i = i[(i + 1) % line != 0]
        w = rng.uniform(-1, 1, len(i))
        row += [i, i + o]
        col += [i + o, i]
        val += [w, w]
    row, col, val = np.concatenate(row), np.concatenate(col), np.concatenate(val)
    o = np.lexsort((col, row))
    rp = np.searchsorted(row[o], np.arange(n + 1)).astype(np.int32)
    return rp, col[o].astype(np.int32), val[o]


# name: (matrix, most block levels a sweep may have, None: as it comes)
MATS = {"lines_31": (W.poisson2d(31, 31)[1:], 31),
        "lines_32": (W.poisson2d(32, 32)[1:], 32),
        "lines_33": (W.poisson2d(33, 33)[1:], 34),
        "lines_65": (W.poisson2d(65, 65)[1:], 67),
        "lines_3": (W.poisson2d(3, 40)[1:], None),
        "lines_40_of_3": (W.poisson2d(40, 3)[1:], None),
        "cube_17": (W.poisson3d(17)[1:], 33),
        "cube_33": (W.poisson3d(33)[1:], 66),
        "grid_251": (W.poisson2d(251, 251)[1:], 258),
        # a block's first row has four entries before its block, the one in its
        # line among them (on one cluster), or five (not); the solutions are
        # past a single CTA's shared memory in both precisions
        "four_outside": (banded(60000, [1, 300, 600, 900], 300)[:], None),
        "five_outside": (banded(60000, [1, 300, 600, 900, 1200], 300)[:], None),
        "permuted": (permuted(*W.poisson2d(30, 30)[1:], 5), None)}
ON_CLUSTER = ("cube_33", "grid_251", "four_outside")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("name", sorted(MATS))
def test_odd_lines(handle, restatement, name, dtype):
    import torch
    from monolish_b200 import device as D
    (rp, ci, v), most = MATS[name]
    v = v.astype(dtype)
    n = len(rp) - 1
    A = D.Crs(handle, n, n, rp, ci, v)
    r = np.random.default_rng(3).uniform(-1, 1, n).astype(dtype)
    for kind in (SOR, IC, ILU):
        pc = D.Precond(A, kind, omega=1.9)
        lower, upper, blocks = pc.info()
        assert blocks >= (n + 31) // 32
        assert pc.sweep_ctas() == ((16, 16) if name in ON_CLUSTER else (0, 0))
        if most is not None:
            assert max(lower, upper) <= most, (lower, upper)
        want_f, _ = restatement.precond_factor(rp, ci, v, kind, omega=1.9)
        assert np.array_equal(pc.factor().cpu().numpy(), want_f)
        z = torch.zeros(n, dtype=torch.float64 if dtype == np.float64 else torch.float32,
                        device="cuda")
        pc.apply(torch.from_numpy(r).cuda(), z)
        want = restatement.precond_apply(rp, ci, v, kind, r, omega=1.9)
        err = np.abs(z.cpu().numpy() - want).max() / np.abs(want).max()
        assert err < (1e-12 if dtype == np.float64 else 1e-5), (kind, err)
        pc.close()
    A.close()


def host_blocks(rp, ci):
    """Blocks cut at 32 rows and where a row and the one before it do not
    depend on each other."""
    n = len(rp) - 1
    rows = np.repeat(np.arange(n), np.diff(rp))
    linked = np.zeros(n + 1, bool)
    linked[rows[ci == rows - 1]] = True
    linked[rows[ci == rows + 1] + 1] = True
    blocks, rows_in = 0, 32
    for i in range(n):
        if rows_in == 32 or not linked[i]:
            blocks, rows_in = blocks + 1, 0
        rows_in += 1
    return blocks


@pytest.mark.parametrize("line,lines", [(33, 61), (40, 50), (63, 9)])
def test_blocks_of_uneven_rows(handle, line, lines):
    """Links between rows are found whatever the rows' lengths are: every
    seventh row also has entries in the first line's columns, and the last
    warp has rows past the end."""
    from monolish_b200 import device as D
    _, rp, ci, v = W.poisson2d(line, lines)
    n = len(rp) - 1
    rng = np.random.default_rng(2)
    cols = [ci[rp[i]:rp[i + 1]] for i in range(n)]
    for i in range(2 * line, n, 7):
        cols[i] = np.union1d(cols[i], rng.choice(line, int(rng.integers(1, line)), replace=False))
    rp = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    ci = np.concatenate(cols).astype(np.int32)
    A = D.Crs(handle, n, n, rp, ci, np.where(np.repeat(np.arange(n), np.diff(rp)) == ci, 99.0, -1))
    for _ in range(3):
        pc = D.Precond(A, SOR, omega=1.0)
        assert pc.info()[2] == host_blocks(rp, ci)
        pc.close()
    A.close()


@pytest.mark.parametrize("kind,plain", [(SOR, True), (ILU, True), (IC, False)])
def test_blocks_weigh_both_sweeps(handle, restatement, kind, plain):
    """Lines of 49 rows below the diagonal, row i + 2 above it: cut blocks save
    the lower sweep 21 levels of scans and cost the upper one 18 levels of
    chains, which weigh three times as much.  An IC factor sweeps the lower
    triangle both ways and takes the cut blocks."""
    from monolish_b200 import device as D
    line, lines = 49, 40
    n = line * lines
    _, rp, ci, v = W.poisson2d(line, lines)
    rows = np.repeat(np.arange(n), np.diff(rp))
    low = ci <= rows
    i = np.arange(n - 2)
    row, col = np.concatenate([rows[low], i]), np.concatenate([ci[low], i + 2])
    val = np.concatenate([v[low], np.full(n - 2, -0.5)])
    o = np.lexsort((col, row))
    rp = np.searchsorted(row[o], np.arange(n + 1)).astype(np.int32)
    ci, v = col[o].astype(np.int32), val[o]
    A = D.Crs(handle, n, n, rp, ci, v)
    pc = D.Precond(A, kind, omega=1.0)
    lower, upper, blocks = pc.info()
    if plain:
        assert (blocks, lower, upper) == (-(-n // 32), 62, 62)
    else:
        assert (blocks, lower, upper) == (host_blocks(rp, ci), 41, 41)
    pc.close()
    A.close()


def test_cluster_sweeps_repeat(handle):
    """258 levels of fewer blocks than CTAs: CTAs without a block in a level
    run ahead of the others.  300 applies give the same bits."""
    import torch
    from monolish_b200 import device as D
    (rp, ci, v), _ = MATS["grid_251"]
    n = len(rp) - 1
    A = D.Crs(handle, n, n, rp, ci, v)
    pc = D.Precond(A, SOR, omega=1.9)
    assert pc.sweep_ctas() == (16, 16)
    r = torch.from_numpy(np.random.default_rng(3).uniform(-1, 1, n)).cuda()
    z = [torch.zeros_like(r) for _ in range(301)]
    for out in z:
        pc.apply(r, out)
    assert all(torch.equal(z[0], out) for out in z)
    pc.close()
    A.close()
