"""The crossover on every blocked side (the Fourier-space children's parents
stay in the passes there), a run-time side, and both kinds of children in one
call, against the oracle.

As in test_gpu_population.py: at most 0.5% of the pixels differ (a crossmap
cell boundary within float rounding of a pixel), elsewhere densities agree
within 1e-4 of the largest."""
import numpy as np
import pytest

from oracle import spring_oracle as o
from s_spi_spring_gb300 import _lib
from test_gpu_population import population

pytestmark = pytest.mark.gpu

CASES = [(256, 1.0, 0.0, True), (256, 0.5, 0.4, False), (384, 0.5, -0.5, True), (512, 0.5, 0.0, False),
         (512, 1.0, 0.7, True), (768, 1.0, -0.3, True), (1024, 0.6, 0.5, True), (2048, 1.0, 0.0, True),
         (100, 0.5, 0.5, True), (64, 1.0, 0.0, False)]


@pytest.mark.parametrize("n,crossft,use_average,update_support", CASES)
def test_crossover_sides(n, crossft, use_average, update_support):
    P = 6 if n <= 512 else 4
    A, rhos, Ss = population(n, P, seed=n)
    errors = np.random.default_rng(n).uniform(0.1, 0.9, P).astype(np.float32)
    best = int(np.argmin(errors))
    avg_d, avg_s = o.get_average(list(rhos), list(Ss), errors, 0.8)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(A)
    e.seed(n)
    e.reserve(2 * P + 2)
    e.upload(0, rhos, Ss)
    e.upload(P, rhos[best][None], Ss[best][None])
    e.upload(P + 1, avg_d[None], avg_s[None])
    e.crossover(0, P, errors, P, P + 1, P + 2, 0.6, 0.4, 1.0, crossft, False, use_average, update_support,
                0.0, 0.0, 2.0)
    gd, gs = e.download(P + 2, P)
    ref = o.crossover_population(list(rhos), list(Ss), errors, Ss[best], avg_d, A, o.ContextRNG(n), 0.6, 0.4,
                                 1.0, crossft, False, use_average, update_support, 0.0, 0.0, 2.0)
    for i, (rd, rs) in enumerate(ref):
        assert np.mean(gs[i] != rs) <= 5e-3, i
        bad = np.abs(gd[i] - rd) > 1e-4 * np.abs(rd).max()
        assert bad.mean() <= 5e-3, (i, bad.mean())
    parents, _ = e.download(0, P)
    assert np.array_equal(parents.view(np.uint32), rhos.view(np.uint32))
