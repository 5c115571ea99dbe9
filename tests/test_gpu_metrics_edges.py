"""Evaluation and alignment on the blocked scratch and on run-time sides:
every side with its own tile shape, more partials per individual than one
reduction chunk (1024, 2048), one pattern per individual, densities full of
zeros of both signs, and an empty density (whose symmetry is not a number).

Tolerance: a float32 transform is good to about log2(n^2) 2^-24 = 1.3e-6 of
its norm, and the metrics compared are no smaller than 1/50 of the terms they
are sums of: 1e-4.
"""
import numpy as np
import pytest

from oracle import spring_oracle as o
from s_spi_spring_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu

KEYS = ("error_fourier", "error_real", "reality", "modulesum", "complexsum", "symmetry")


@pytest.mark.parametrize("n", [16, 50, 128, 256, 384, 512, 768, 1024, 2048])
def test_evaluate_and_reshift(n):
    P = 3 if n <= 512 else 2
    rng = np.random.default_rng(n)
    amps, rhos, Ss = [], [], []
    for k in range(P):
        I, obj, supp = synthetic.polygon_pattern(seed=k + 1, n=n, diameter=n * 0.3, photons=1e7, stop_radius=1)
        amps.append(_lib.prepare_pattern(I, (-1, -1), True))
        noise = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        r = np.roll(obj * np.exp(1j) + 0.02 * noise * supp, (2 * k, -k), axis=(0, 1))
        s = np.roll(supp, (2 * k, -k), axis=(0, 1)).astype(np.int32)
        # zeros of both signs outside
        sign = rng.integers(0, 2, (2, n, n)) * 2 - 1
        r = np.where(r == 0, 0.0 * sign[0] + 1j * (0.0 * sign[1]), r).astype(np.complex64)
        rhos.append(r)
        Ss.append(s)
    rhos, Ss = np.stack(rhos), np.stack(Ss)
    for patterns in (1, P):
        e = _lib.Engine(n, 0)
        if patterns == 1:
            e.set_amplitudes(amps[0])
        else:
            e.set_amplitudes_batch(np.stack(amps), 1)
        e.upload(0, rhos, Ss)
        for i, m in enumerate(e.evaluate(0, P)):
            ref = o.evaluate(rhos[i].astype(complex), Ss[i], amps[0] if patterns == 1 else amps[i])
            for k in KEYS:
                assert abs(m[k] - ref[k]) <= 1e-4 * max(abs(ref[k]), 0.02), (i, k, m[k], ref[k])
    e = _lib.Engine(n, 0)
    e.set_amplitudes(amps[0])
    e.upload(0, rhos, Ss)
    e.reshift(0, P, -1, rhos[0], 0.0, 2.0)
    got, gs = e.download(0, P)
    for i in range(P):
        rr, rs = o.reshift(rhos[i].astype(complex), Ss[i], rhos[0].astype(complex), amps[0], 0.0, 2.0)
        assert np.array_equal(gs[i], rs), i
        assert np.linalg.norm(got[i] - rr) / np.linalg.norm(rr) < 1e-5, i


@pytest.mark.parametrize("n", [50, 128, 256])
def test_empty_density(n):
    I, obj, supp = synthetic.polygon_pattern(seed=1, n=n, diameter=n * 0.3, photons=1e7, stop_radius=1)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(_lib.prepare_pattern(I, (-1, -1), True))
    e.upload(0, np.stack([np.zeros((n, n), np.complex64), obj.astype(np.complex64)]), np.stack([supp, supp]).astype(np.int32))
    m = e.evaluate(0, 2)
    assert np.isnan(m[0]["symmetry"]) and m[0]["modulesum"] == 0.0 and m[0]["error_fourier"] == 1.0
    assert 0.0 < m[1]["symmetry"] <= 1.0 + 1e-4
