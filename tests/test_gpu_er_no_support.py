"""Error reduction of individuals without any support among others, in
populations large enough for the live row tiles: bit for bit the row-major
passes' result, by any number of iterations.  (The density becomes zeros of
either sign, and the modulus projection of an all-zero transform goes by their
signs.)"""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib, synthetic
from test_gpu_er_live import ROW_MAJOR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", sorted(ROW_MAJOR))
def test_no_support(n):
    P = max(4, -(-(1 << 22) // (n * n)))
    rng = np.random.default_rng(n)
    I, _, _ = synthetic.polygon_pattern(seed=2, n=n, diameter=n * 0.23, photons=1e7, stop_radius=max(2, n // 64))
    S = np.zeros((P, n, n), np.int32)
    for k in range(P):
        if k % 3 == 1:
            S[k, n // 3:n // 2, n // 4:n // 2] = 1
        elif k % 3 == 2:
            S[k, n - 1, 0] = -2
    dens = (rng.standard_normal(S.shape) + 1j * rng.standard_normal(S.shape)).astype(np.complex64)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(_lib.prepare_pattern(I, (-1, -1), True))
    for iters in (1, 2, 3, 6):
        out = []
        for tiles in (ROW_MAJOR[n], (0, 0)):
            e.upload(0, dens, S)
            e.set_tiles(*tiles)
            e.er(0, P, iters, 0.0)
            out.append(e.download(0, P)[0])
        for k in range(P):
            assert np.array_equal(out[0][k], out[1][k]), (iters, k)
