"""Error reduction through the support's row tiles (blocked sides) against the
row-major passes, which run every row: bit-identical for supports that are
empty, one pixel, at the tile edges, scattered, full, and other than 0 / 1, each
in its own individual; a density that is not finite stays so, also where its
support is empty."""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu
ROW_MAJOR = {256: (8, 8), 384: (16, 2), 512: (8, 4), 768: (8, 1), 1024: (8, 1), 2048: (4, 1)}


@pytest.mark.parametrize("n", sorted(ROW_MAJOR))
def test_er_supports(n):
    rng = np.random.default_rng(n)
    I, _, _ = synthetic.polygon_pattern(seed=2, n=n, diameter=n * 0.23, photons=1e7, stop_radius=max(2, n // 64))
    S = np.zeros((6, n, n), np.int32)
    S[1, n - 1, 0] = 1
    S[2, [0, 3, 4, n // 2, n - 4], :] = 1
    S[3] = rng.integers(0, 60, (n, n)) == 0
    S[4] = 1
    S[5, n // 3:n // 2, n // 4:n // 2] = rng.integers(-2, 4, (n // 2 - n // 3, n // 2 - n // 4))
    dens = (rng.standard_normal(S.shape) + 1j * rng.standard_normal(S.shape)).astype(np.complex64)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(_lib.prepare_pattern(I, (-1, -1), True))
    for first, count, iters, reality in ((0, 6, 3, 0.0), (1, 4, 1, 0.4), (0, 6, 0, 0.0), (4, 1, 2, 0.0)):
        out = []
        for tiles in (ROW_MAJOR[n], (0, 0)):
            e.upload(0, dens, S)
            e.set_tiles(*tiles)
            e.er(first, count, iters, reality)
            out.append(e.download(0, 6)[0])
        assert np.array_equal(out[0], out[1]), (first, iters)
    dens[0, 7, 9] = np.nan
    dens[5, 3, 2] = np.inf
    e.upload(0, dens, S)
    e.set_tiles(0, 0)
    e.er(0, 6, 2, 0.0)
    got = e.download(0, 6)[0]
    assert np.isnan(got[0]).all() and np.isnan(got[5]).all() and np.isfinite(got[1:5]).all()
