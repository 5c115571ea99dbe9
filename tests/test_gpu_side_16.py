"""The smallest compiled side: every update, the metrics and the shrink-wrap at
16 against the oracle (one iteration: the tolerance of test_gpu_any_side.py for
sides of this size), alone and in a population."""
import numpy as np
import pytest

from oracle import spring_oracle as o
from s_spi_spring_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P", [1, 7, 300])
def test_iterations_at_16(P):
    n = 16
    rng = np.random.default_rng(P)
    A = (np.abs(rng.standard_normal((n, n))) + 0.5).astype(np.float32)
    A[3, 4] = -1.0
    dens = (rng.standard_normal((P, n, n)) + 1j * rng.standard_normal((P, n, n))).astype(np.complex64)
    S = rng.integers(0, 2, (P, n, n)).astype(np.int32)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(A)
    for alg, beta in (("hio", 0.9), ("raar", 0.87), ("er", None)):
        e.upload(0, dens, S)
        args = (0, P, 1) if beta is None else (0, P, 1, beta)
        getattr(e, alg)(*args)
        got, _ = e.download(0, P)
        for i in range(0, P, 41):
            d = dens[i].astype(complex)
            ref = o.er(d, S[i], A, 1, 0.0) if beta is None else getattr(o, alg)(d, S[i], A, 1, beta, 0.0)
            assert np.linalg.norm(got[i] - ref) <= 5e-6 * np.linalg.norm(ref), (alg, i)
    assert np.isfinite([m["error"] for m in e.evaluate(0, P)]).all()
