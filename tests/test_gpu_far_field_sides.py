"""The far field and the average module of a population at every compiled side
against 64-bit transforms, per individual: a transform of 2 log2 n radix-2
stages rounds to about 2 log2(n) 2^-24 of the norm (1.3e-6 at 2048), 5e-6 here."""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 32, 64, 128, 256, 384, 512, 768, 1024, 2048, 100])
def test_far_field(n):
    P = 3
    rng = np.random.default_rng(n)
    dens = (rng.standard_normal((P, n, n)) + 1j * rng.standard_normal((P, n, n))).astype(np.complex64)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(np.ones((n, n), np.float32))
    e.upload(0, dens, np.ones((P, n, n), np.int32))
    want = np.abs(np.fft.ifft2(dens.astype(complex)) * n * n)
    got = e.far_field(1, 2)
    for i in range(2):
        assert np.linalg.norm(got[i] - want[1 + i]) <= 5e-6 * np.linalg.norm(want[1 + i])
    mean = e.average_module(0, P, np.zeros(P, np.float32), True, 1.0)
    assert np.linalg.norm(mean - want.mean(axis=0)) <= 5e-6 * np.linalg.norm(want.mean(axis=0))
