"""The tile and thread rules of the sides without a compiled plan: one
individual (tiles narrowed to fill the GPU) and many of them (whole tiles),
the same bits individual by individual; every radix of a pass, alone and with
a larger prime, and a run-time prime with one, two and four butterflies per
thread, against the oracle (tolerance of test_gpu_any_side.py)."""
import numpy as np
import pytest

from oracle import spring_oracle as o
from s_spi_spring_gb300 import _lib, synthetic
from test_gpu_any_side import case, rel, tol1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 5, 6, 7, 9, 10, 18, 37, 45, 54, 60, 90, 100, 101, 190, 202, 270, 303, 420, 606, 630])
def test_one_iteration_and_tile_widths(n):
    if n < 18:
        rng = np.random.default_rng(n)
        A = np.abs(rng.standard_normal((n, n))).astype(np.float32) + 0.5
        dens = (rng.standard_normal((2, n, n)) + 1j * rng.standard_normal((2, n, n))).astype(np.complex64)
        S = rng.integers(0, 2, (2, n, n)).astype(np.int32)
    else:
        A, dens, S = case(n, 2, seed=n)[:3]
    many = max(3, int(400 * 8 / n) + 1)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(A)
    reps = (many + 1) // 2
    e.upload(0, np.concatenate([dens] * reps), np.concatenate([S] * reps))
    e.raar(0, 2 * reps, 1, 0.9, 0.0)
    got, _ = e.download(0, 2 * reps)
    for k in range(0, 2 * reps, 2):
        assert np.array_equal(got[k:k + 2].view(np.uint32), got[:2].view(np.uint32))
    for i in range(2):
        e.upload(0, dens[i][None], S[i][None])
        e.raar(0, 1, 1, 0.9, 0.0)
        one, _ = e.download(0, 1)
        assert np.array_equal(one[0].view(np.uint32), got[i].view(np.uint32))
        assert rel(got[i], o.raar(dens[i].astype(complex), S[i], A, 1, 0.9, 0.0)) < 5e-6
