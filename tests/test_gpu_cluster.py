"""One cluster per individual (the default of small sides) against the pass
kernels (explicit tile codes): the same arithmetic per element, so the results
are bit-identical -- supports other than 0 / 1, one pattern per individual, a
range inside the population, no iterations, a phase gate, more individuals than
fit the GPU at once, and on both sides of the rule's limit."""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu


def run(e, tiles, first, count, alg, iters, reality, dens, S):
    e.upload(0, dens, S)
    e.set_tiles(*tiles)
    if alg == "er":
        e.er(first, count, iters, reality)
    else:
        getattr(e, alg)(first, count, iters, 0.9, reality)
    return e.download(0, len(dens))[0]


@pytest.mark.parametrize("n", [32, 64, 128])
def test_bit_identical_to_passes(n):
    P = 5
    rng = np.random.default_rng(n)
    amps = []
    for k in range(P):
        I, _, _ = synthetic.polygon_pattern(seed=k, n=n, diameter=n * 0.3, photons=1e7, stop_radius=2)
        amps.append(_lib.prepare_pattern(I, (-1, -1), True))
    dens, S = synthetic.start_population(n, P, n * 0.25, seed=3)
    S[1] *= 2
    S[2, n // 2, n // 2] = -1
    S[3, 5, :] = rng.integers(0, 3, n)
    e = _lib.Engine(n, 0)
    for patterns in (1, P):
        if patterns == 1:
            e.set_amplitudes(amps[0])
        else:
            e.set_amplitudes_batch(np.stack(amps), 1)
        for alg in ("hio", "raar", "er"):
            for first, count, iters, reality in ((0, P, 3, 0.0), (1, 3, 2, 0.4), (2, 1, 0, 0.0)):
                a = run(e, (16, 8), first, count, alg, iters, reality, dens, S)
                b = run(e, (0, 0), first, count, alg, iters, reality, dens, S)
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (patterns, alg, first, iters)


@pytest.mark.parametrize("n,P", [(32, 700), (64, 400), (128, 48), (128, 49)])
def test_many_individuals(n, P):
    I, _, _ = synthetic.polygon_pattern(seed=1, n=n, diameter=n * 0.3, photons=1e7, stop_radius=2)
    dens, S = synthetic.start_population(n, 7, n * 0.25, seed=5)
    reps = -(-P // 7)
    dens, S = np.concatenate([dens] * reps)[:P], np.concatenate([S] * reps)[:P]
    e = _lib.Engine(n, 0)
    e.set_amplitudes(_lib.prepare_pattern(I, (-1, -1), True))
    a = run(e, (16, 8), 0, P, "raar", 2, 0.0, dens, S)
    b = run(e, (0, 0), 0, P, "raar", 2, 0.0, dens, S)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_autotune_may_keep_the_default():
    """At a side whose default is a cluster per individual the tuner compares it
    with the codes it times, and the densities come back as they were."""
    n, P = 64, 6
    I, _, _ = synthetic.polygon_pattern(seed=1, n=n, diameter=n * 0.3, photons=1e7, stop_radius=2)
    dens, S = synthetic.start_population(n, P, n * 0.25, seed=5)
    e = _lib.Engine(n, 0)
    e.set_amplitudes(_lib.prepare_pattern(I, (-1, -1), True))
    before = run(e, (16, 8), 0, P, "raar", 3, 0.0, dens, S)
    e.upload(0, dens, S)
    e.autotune(0, P)
    assert np.array_equal(e.download(0, P)[0].view(np.uint32), dens.view(np.uint32))
    e.raar(0, P, 3, 0.9, 0.0)
    assert np.array_equal(e.download(0, P)[0].view(np.uint32), before.view(np.uint32))
