"""Gathering individuals (spe_gather) at odd sides, whose individuals start on
any 8-byte boundary (density) and 4-byte boundary (support), and at even ones:
every pixel of both arrays arrives, and nothing else is written."""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 50, 63, 64, 101, 256])
def test_gather(n):
    P = 9
    rng = np.random.default_rng(n)
    dens = (rng.standard_normal((P, n, n)) + 1j * rng.standard_normal((P, n, n))).astype(np.complex64)
    S = rng.integers(-3, 100, (P, n, n)).astype(np.int32)
    e = _lib.Engine(n, 0)
    e.upload(0, dens, S)
    src, first = [8, 1, 1, 0], 3
    e.gather(src, first)
    want_d, want_s = dens.copy(), S.copy()
    want_d[first:first + 4], want_s[first:first + 4] = dens[src], S[src]
    got_d, got_s = e.download(0, P)
    assert np.array_equal(got_d.view(np.uint32), want_d.view(np.uint32))
    assert np.array_equal(got_s, want_s)
