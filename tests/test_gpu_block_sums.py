"""The sums of the reducing passes keep a double's digits: the amplitude loss
of an empty density is the sum of the known amplitudes' squares, here whole
numbers from 1 to 2^50 whose total is below 2^53, so that doubles add them
exactly in any order.  At most one pixel of a thread is known (the first
sixteenth of the rows), and each square is a float: nothing rounds before the
sum."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from s_spi_spring_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 32, 64, 100, 128, 256, 263, 384, 512, 768, 1000, 1024, 2048])
def test_exact_sum(n):
    rng = np.random.default_rng(n)
    rows = n // 16
    A = np.full((n, n), -1.0, np.float32)
    small = rng.integers(1, 10, (rows, n))
    middle = 1024 + rng.integers(1, 256, (rows, n))
    A[:rows] = np.where(rng.random((rows, n)) < 0.6, middle, small)
    for k in range(4):
        A[rng.integers(0, rows), (k * n) // 4] = 2.0 ** 25
    want = int((A[:rows].astype(np.int64) ** 2).sum())
    assert want < 2 ** 53
    e = _lib.Engine(n, 0)
    e.set_amplitudes(A)
    P = 3
    d = torch.zeros(P, n, n, dtype=torch.complex64, device="cuda")
    s = torch.ones(P, n, n, dtype=torch.int32, device="cuda")
    g, loss = torch.empty_like(d), torch.empty(2, P, dtype=torch.float64, device="cuda")
    e.set_stream(torch.cuda.current_stream().cuda_stream or 1)
    e.loss_grad(d.data_ptr(), s.data_ptr(), P, 0, 0.0, loss[0].data_ptr())
    e.loss_grad(d.data_ptr(), s.data_ptr(), P, 0, 0.0, loss[1].data_ptr(), g.data_ptr())
    torch.cuda.synchronize()
    assert loss.flatten().tolist() == [float(want)] * (2 * P)
