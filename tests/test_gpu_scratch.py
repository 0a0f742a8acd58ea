"""Calls whose scratch memory cannot be had go to the kernels that need less of
it instead of failing.  The device's pool is exchanged for one of 32 MiB (the
smallest there is), part of it held; nothing else runs out."""
import contextlib

import numpy as np
import pytest

from monolish_b200 import _abi
from monolish_b200 import workloads as W

pytestmark = pytest.mark.gpu
MIB = 1 << 20


@contextlib.contextmanager
def small_pool(held):
    """A handle whose allocations come from a 32-MiB pool with `held` bytes
    taken."""
    from monolish_b200 import device as D
    rt = pytest.importorskip("cuda.bindings.runtime")

    def ok(result):
        assert int(result[0]) == 0, result[0]
        return result[1] if len(result) > 1 else None
    props = rt.cudaMemPoolProps()
    props.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
    props.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
    props.location.id = 0
    props.maxSize = 32 * MIB
    before = ok(rt.cudaDeviceGetMemPool(0))
    pool = ok(rt.cudaMemPoolCreate(props))
    block = ok(rt.cudaMallocFromPoolAsync(held, pool, 0)) if held else None
    ok(rt.cudaDeviceSetMemPool(0, pool))
    h = D.Handle()
    try:
        yield h
    finally:
        h.close()
        ok(rt.cudaDeviceSetMemPool(0, before))
        if block is not None:
            ok(rt.cudaFreeAsync(block, 0))
        ok(rt.cudaStreamSynchronize(0))
        ok(rt.cudaMemPoolDestroy(pool))


def solve(A, n, **kw):
    import torch
    from monolish_b200 import device as D
    b = torch.ones(n, dtype=torch.float64, device="cuda")
    x = torch.zeros_like(b)
    r = D.cg_solve(A, b, x, 1e-6 * np.sqrt(n), 5000, **kw)
    y = torch.empty_like(b)
    A.matvec(x, y)
    return r.status, float(torch.linalg.vector_norm(b - y)) / np.sqrt(n)


@pytest.mark.parametrize("engine,held", [(_abi.ENGINE_CLUSTER, 24 * MIB), (_abi.ENGINE_GRID, 0)])
def test_cg_without_slices(cuda, engine, held):
    """131,072 rows at 8,192 a CTA stream 10 MiB of slices (vectors: 2 MiB);
    80^3 rows on the whole GPU 47 MiB (vectors: 16 MiB)."""
    from monolish_b200 import device as D
    n, rp, ci, v = W.poisson2d(512, 256) if held else W.poisson3d(80)
    v[np.repeat(np.arange(n), np.diff(rp)) == ci] += 0.5
    with small_pool(held) as h:
        A = D.Crs(h, n, n, rp, ci, v)
        status, left = solve(A, n, engine=engine)
        A.close()
    assert status == 0 and left < 1.01e-6


def test_batch_without_slices(cuda):
    """150 systems of one CTA each stream 74 MiB of slices."""
    import torch
    from monolish_b200 import device as D
    n, rp, ci, v = W.poisson2d(128, 64)
    v[np.repeat(np.arange(n), np.diff(rp)) == ci] += 0.5
    with small_pool(0) as h:
        B = D.Batch(h, [(rp, ci, v)] * 150)
        b = torch.ones(150 * n, dtype=torch.float64, device="cuda")
        x = torch.zeros_like(b)
        status, _, resid = B.solve("cg", b, x, 1e-6, 5000)
        B.close()
    assert (status == 0).all() and (resid < 1e-6).all()
    assert torch.equal(x[:n], x[-n:])


def test_coo_sort_without_groups(cuda, restatement):
    """700,000 entries in 2,800,000 rows: 34 MiB of groups, 28 MiB for the
    general sort."""
    import torch
    from monolish_b200 import device as D
    rng = np.random.default_rng(5)
    k, rows = 700000, 2800000
    row, col = (rng.integers(0, m, k, dtype=np.int32) for m in (rows, 1000))
    val = rng.uniform(-1, 1, k)
    d = [torch.from_numpy(a).cuda() for a in (row, col, val)]
    with small_pool(0) as h:
        cnt = D.coo_sort(h, rows, 1000, *d, merge=True)
    er, ec, ev = restatement.coo_sort(row, col, val, True)
    assert cnt == len(er)
    for got, want in zip(d, (er, ec, ev)):
        assert np.array_equal(got.cpu().numpy()[:cnt], want)
