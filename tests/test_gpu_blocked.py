"""The blocked-scratch iteration kernels (the default where a side has them)
against the row-major ones: the same arithmetic per element, so the results
are bit-identical -- also where the support is not 0 / 1 (read as integers by
the tiles that hold such pixels), with one pattern per individual, and on a
range that starts inside the population."""
import numpy as np
import pytest

from s_spi_spring_gb300 import _lib, synthetic

pytestmark = pytest.mark.gpu

ROW_MAJOR = {256: (8, 8), 384: (16, 2), 512: (8, 4), 768: (8, 1), 1024: (8, 1), 2048: (4, 1)}


def call(e, alg, first, count, iters, reality):
    if alg == "er":
        e.er(first, count, iters, reality)
    else:
        getattr(e, alg)(first, count, iters, 0.9, reality)


@pytest.mark.parametrize("n", sorted(ROW_MAJOR))
def test_blocked_scratch_bit_identical(n):
    P = 5 if n <= 1024 else 3
    rng = np.random.default_rng(n)
    amps = []
    for k in range(P):
        I, _, _ = synthetic.polygon_pattern(seed=k, n=n, diameter=n * 0.23, photons=1e7, stop_radius=max(2, n // 64))
        amps.append(_lib.prepare_pattern(I, (-1, -1), True))
    dens, S = synthetic.start_population(n, P, n * 0.2, seed=3)
    S[1] *= 2                          # uniform, but not 0 / 1
    S[2, n // 2, n // 2] = -1          # one row tile of one individual
    S[2, 5, :] = rng.integers(0, 3, n)
    e = _lib.Engine(n, 0)
    for patterns in (1, P):
        if patterns == 1:
            e.set_amplitudes(amps[0])
        else:
            e.set_amplitudes_batch(np.stack(amps), 1)
        for alg, iters, reality in (("raar", 3, 0.0), ("hio", 2, 0.5), ("er", 2, 0.5), ("raar", 0, 0.0)):
            out = []
            for tiles in (ROW_MAJOR[n], (0, 0)):
                e.set_tiles(*tiles)
                e.upload(0, dens, S)
                call(e, alg, 1, P - 1, iters, reality)
                out.append(e.download(0, P)[0])
            assert np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32)), (alg, patterns)
            assert np.array_equal(out[1][0], dens[0])


def test_blocked_codes_go_together():
    e = _lib.Engine(512, 0)
    c, r = e.tiles()
    assert c > 800 and r > 800
    e.set_tiles(c, r)
    e.set_tiles(c, 0)
    assert e.tiles() == (c, r)
    for bad in ((c, 4), (8, r)):
        with pytest.raises(_lib.EngineError):
            e.set_tiles(*bad)
    e.set_tiles(8, 0)
    assert e.tiles() == (8, 4)
