"""A crossover of several hundred individuals (its workspace grows with each
one), with and without the average, against the oracle: the tolerances of
test_gpu_population.py, on the average of the children and for 98% of them (a
crossmap whose cell boundary runs along a row of pixels may cost a child
more)."""
import numpy as np
import pytest

from oracle import spring_oracle as o
from s_spi_spring_gb300 import _lib
from test_gpu_population import population

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,use_average", [(400, 0.0), (600, 0.5)])
def test_crossover_many(P, use_average):
    n = 64
    A, rhos, Ss = population(n, 6, seed=n)
    rhos, Ss = np.concatenate([rhos] * (P // 6 + 1))[:P], np.concatenate([Ss] * (P // 6 + 1))[:P]
    errors = np.random.default_rng(P).uniform(0.1, 0.9, P).astype(np.float32)
    best = int(np.argmin(errors))
    avg_d, avg_s = o.get_average(list(rhos), list(Ss), errors, 0.8)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(A)
    e.seed(P)
    e.reserve(2 * P + 2)
    e.upload(0, rhos, Ss)
    e.upload(P, rhos[best][None], Ss[best][None])
    e.upload(P + 1, avg_d[None], avg_s[None])
    e.crossover(0, P, errors, P, P + 1, P + 2, 0.6, 0.4, 1.0, 0.5, False, use_average, True, 0.0, 0.0, 2.0)
    gd, gs = e.download(P + 2, P)
    ref = o.crossover_population(list(rhos), list(Ss), errors, Ss[best], avg_d, A, o.ContextRNG(P), 0.6, 0.4,
                                 1.0, 0.5, False, use_average, True, 0.0, 0.0, 2.0)
    wrong_s = np.array([np.mean(s != rs) for s, (_, rs) in zip(gs, ref)])
    wrong_d = np.array([np.mean(np.abs(d - rd) > 1e-4 * np.abs(rd).max()) for d, (rd, _) in zip(gd, ref)])
    for wrong in (wrong_s, wrong_d):
        assert wrong.mean() <= 5e-3 and np.mean(wrong > 5e-3) <= 0.02, (wrong.mean(), np.flatnonzero(wrong > 5e-3))
