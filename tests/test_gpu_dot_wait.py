"""dot / nrm2 returned to the host: the results of many waits in a row, of two
handles on streams of their own in two threads, behind unfinished work, and of
non-finite sums."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float64", "float32"])
@pytest.mark.parametrize("n", [0, 1, 255, 1025, 16383, 3000001])
def test_values_behind_pending_work(handle, n, dtype):
    import torch
    x = torch.rand(n, dtype=getattr(torch, dtype), device="cuda") - 0.5
    y = torch.ones_like(x)
    for k in range(1, 4):
        handle.axpy(1.0, x, y)  # y = 1 + k x, possibly still running
        want = float((x.double() * y.double()).sum())
        scale = float((x.double() * y.double()).abs().sum())
        assert abs(handle.dot(x, y) - want) <= 1e-14 * scale
    assert abs(handle.nrm2(x) - float(torch.linalg.vector_norm(x.double()))) <= 1e-14 * max(1, n)


def test_non_finite(handle):
    import torch
    x = torch.ones(5000, dtype=torch.float64, device="cuda")
    x[17] = float("inf")
    assert handle.nrm2(x) == np.inf
    x[18] = float("nan")
    assert np.isnan(handle.dot(x, x))


def test_two_handles_two_threads(cuda):
    import torch
    from monolish_b200.device import Handle
    bad = []

    def work(seed):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            h = Handle()
            x = torch.full((20000 + seed,), float(seed), dtype=torch.float64, device="cuda")
            for _ in range(300):
                if h.dot(x, x) != float(seed) ** 2 * (20000 + seed):
                    bad.append(seed)
            h.close()
    threads = [threading.Thread(target=work, args=(k,)) for k in (2, 3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
