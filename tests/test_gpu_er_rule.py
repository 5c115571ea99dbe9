"""Error reduction on both sides of the rule that turns the live row tiles on
(more than 2^21 pixels), with supports over few rows (the list is used) and over most
(every tile runs), at every blocked side, against the row-major passes: bit for
bit, in the whole population and in a range inside it, with one iteration and
without any; and a density that is not finite where there is no support."""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib, synthetic
from test_gpu_er_live import ROW_MAJOR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", ["few", "most", "mixed"])
@pytest.mark.parametrize("n", sorted(ROW_MAJOR))
def test_er_rule(n, rows):
    rng = np.random.default_rng(n)
    limit = (2 << 20) // (n * n) + 1  # the smallest population with the list
    P = limit + 2
    I, _, _ = synthetic.polygon_pattern(seed=2, n=n, diameter=n * 0.23, photons=1e7, stop_radius=max(2, n // 64))
    S = np.zeros((P, n, n), np.int32)
    for k in range(P):
        kind = {"few": k % 3, "most": 3 + k % 2, "mixed": k % 5}[rows]
        if kind == 1:
            S[k, [0, 3, 4, n // 2, n - 4], :] = 1
        elif kind == 2:
            S[k, n // 3:n // 2, n // 4:n // 2] = rng.integers(-2, 4, (n // 2 - n // 3, n // 2 - n // 4))
        elif kind == 3:
            S[k] = rng.integers(0, 60, (n, n)) == 0
        elif kind == 4:
            S[k] = 1
    dens = (rng.standard_normal(S.shape) + 1j * rng.standard_normal(S.shape)).astype(np.complex64)
    if rows == "few":
        dens[P - 1, 1, 2] = np.inf  # (a kind without support, or away from it)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(_lib.prepare_pattern(I, (-1, -1), True))
    calls = [(0, P, 3), (1, limit, 2), (2, limit, 1), (0, limit, 0)]
    if limit > 1:
        calls.append((1, limit - 1, 2))  # below the limit
    for first, count, iters in calls:
        out = []
        for tiles in (ROW_MAJOR[n], (0, 0)):
            e.upload(0, dens, S)
            e.set_tiles(*tiles)
            e.er(first, count, iters, 0.0)
            out.append(e.download(0, P)[0].view(np.float32))
        assert np.array_equal(out[0], out[1], equal_nan=True), (first, count, iters)
        if rows == "few" and first + count == P and iters > 0:
            assert np.isnan(out[1][P - 1]).all()
