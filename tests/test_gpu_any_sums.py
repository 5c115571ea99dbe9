"""The metrics' sums at sides without a compiled plan do not depend on how many
pixels of a tile a thread adds: the modulus sum of a density that is 2^25 in
every 32nd row and 1 elsewhere (a float sum drops every 1 that follows a 2^25)
is right to its final rounding, 2^-24 of it, with a factor 2 for the root."""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 40])
@pytest.mark.parametrize("n", [50, 97, 100, 101, 263, 303, 526, 600, 1054])
def test_modulus_sum(n, P):
    P = min(P, 1 + (1 << 22) // (n * n))
    rng = np.random.default_rng(n)
    dens = np.ones((P, n, n), np.complex64)
    dens[:, ::32] = 2.0 ** 25
    # (not a phase of pi, which the evaluation's gate takes out)
    dens *= np.array([1, 1j, -1j], np.complex64)[np.arange(P) % 3][:, None, None]
    e = _lib.Engine(n, 0)
    e.set_amplitudes((np.abs(rng.standard_normal((n, n))) + 0.5).astype(np.float32))
    e.upload(0, dens, np.ones((P, n, n), np.int32))
    want = float(np.abs(dens[0]).astype(np.float64).sum())
    for m in e.evaluate(0, P):
        assert abs(m["modulesum"] - want) <= 2.0 ** -23 * want
